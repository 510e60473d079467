"""The contraction FLOPs that bench.py reports its rates with: what the stage
kernels' layouts hold, counted from the operator shapes of order 4."""
import bench


def test_contraction_flops_of_order_4():
    Np, Nc, Ng, m = 15, 54, 10, 4
    Nf = 3 * Ng
    volume = Nc * Np + 2 * Nc * Np  # V, Dr and Ds
    lift = Nf * Np
    # float64: each side's trace at a face point is a sum over the face's five nodes
    assert bench.contraction_flops("fp64", 4, Np, Nc, Ng, m) == 2 * m * (volume + lift + 2 * Nf * 5) == 25440
    # mixed: the trace GEMM contracts all nodes of the element
    assert bench.contraction_flops("mixed", 4, Np, Nc, Ng, m) == 2 * m * (volume + lift + Nf * Np) == 26640
