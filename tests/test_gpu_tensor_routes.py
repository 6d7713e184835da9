"""The two routes of the scalar-tensor FP64 two-body terms: the products'
(panels and transforms by batches of a j-class, digit products) against the
FP64-pipe kernels, which run where a first call comes under capture and the
products' plans cannot be made.  An element is a few nested sums of at most
600 additions each and |terms| below 25 times the largest element, so the two
agree within 2 x 600 x 2^-53 x 25 < 4e-12 of it; infinities meet the same
elements."""
import numpy as np
import pytest

import imsrg_gb300 as ig
from modelspace_ref import RefModelSpace

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("emax,nucleus,rank,herm", [(1, "O16", (1, 0, 1), 1), (3, "O16", (2, 0, 0), 1), (3, "O18", (0, 1, 0), -1),
                                                    (4, "O16", (3, 1, 1), -1), (2, "O16", (5, 0, 0), 1)])
@pytest.mark.parametrize("term", ["comm222_phst", "comm222_pp_hh_221st"])
@pytest.mark.parametrize("inf", [False, True])
def test_products_vs_fp64_pipe(emax, nucleus, rank, herm, term, inf):
    ref = RefModelSpace(emax, *{"O16": (16, 8), "O18": (18, 8)}[nucleus])
    ms = ig.ModelSpace(emax, nucleus, nucleus)
    X, Y = ref.random_operator(5, True), ref.random_tensor(6, *rank)
    if inf:
        if not np.any(Y):
            pytest.skip("no element of the rank")
        Y[np.flatnonzero(Y)[-1]] = np.inf
    out = []
    with ig.DeviceOperator(ms, 1) as dX, ig.DeviceOperator(ms, herm, rank) as dY:
        dX.upload(X)
        dY.upload(Y)
        for captured in (True, False):
            with ig.DeviceOperator(ms, -1 if herm == 1 else 1, rank) as dZ:
                if captured:
                    st = torch.cuda.Stream()
                    torch.cuda.synchronize()
                    g = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
                        ig.Commutator.device_tensor_term(term, dX, dY, dZ, "fp64", st.cuda_stream)
                    g.replay()
                else:
                    ig.Commutator.device_tensor_term(term, dX, dY, dZ, "fp64")
                torch.cuda.synchronize()
                out.append(dZ.download())
    pipe, prod = out
    fine = np.isfinite(pipe)
    assert np.array_equal(fine, np.isfinite(prod))
    top = np.max(abs(pipe[fine]), initial=0.0)
    assert np.max(abs(pipe[fine] - prod[fine]), initial=0.0) <= 4e-12 * top


@pytest.mark.parametrize("emax,nucleus,rank,herm", [(5, "O16", (2, 0, 0), 1), (5, "O18", (3, 0, 1), -1), (6, "O16", (0, 1, 0), 1)])
@pytest.mark.parametrize("term", ["comm222_phst", "comm222_pp_hh_221st"])
@pytest.mark.parametrize("inf", [False, True])
def test_products_vs_fp64_pipe_above_the_rule(emax, nucleus, rank, herm, term, inf):
    """At sizes from which a call outside a capture takes the products (5e7
    multiply-adds of the ladder, 1e7 of Z bar)."""
    test_products_vs_fp64_pipe(emax, nucleus, rank, herm, term, inf)


@pytest.mark.parametrize("emax,nucleus,rank,herm", [(1, "O16", (1, 1, 0), 1), (2, "O16", (0, 1, 0), 1), (2, "O16", (2, 0, 0), -1), (3, "O18", (2, 0, 0), 1)])
def test_whole_commutator_either_side_of_the_rule(emax, nucleus, rank, herm):
    """Captured (FP64-pipe kernels throughout) against not captured (products
    from 2.5e5 multiply-adds of Z bar): same bound."""
    ref = RefModelSpace(emax, *{"O16": (16, 8), "O18": (18, 8)}[nucleus])
    ms = ig.ModelSpace(emax, nucleus, nucleus)
    X, Y = ref.random_operator(5, True), ref.random_tensor(6, *rank)
    with ig.DeviceOperator(ms, 1) as dX, ig.DeviceOperator(ms, herm, rank) as dY, ig.DeviceOperator(ms, 1, rank) as dZ:
        dX.upload(X)
        dY.upload(Y)
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=st, capture_error_mode="relaxed"):
            ig.Commutator.device_scalar_tensor(dX, dY, dZ, "fp64", st.cuda_stream)
        g.replay()
        torch.cuda.synchronize()
        pipe = dZ.download()
        ig.Commutator.device_scalar_tensor(dX, dY, dZ, "fp64")
        torch.cuda.synchronize()
        prod = dZ.download()
    assert np.max(abs(pipe), initial=0.0) > 0
    assert np.max(abs(pipe - prod)) <= 4e-12 * np.max(abs(pipe))
