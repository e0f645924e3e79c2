"""The tensor-core expectation at the edge of its static shared memory (48 KB):
every shape whose weights, row scales and barrier fit there compiles, whether
or not the row sums and the node bits fit beside them, and its table is right."""

import numpy as np
import pytest

from pylcm_b200.codegen import RegimeKernels, device_header, tc_header
from tests.test_codegen import NVRTC, nvrtc_compile
from tests.test_expectation_gpu import _sum

# (rows, nodes): with sums and bits, with sums only, and with neither
EDGES = [(91, 64), (93, 64), (94, 64), (95, 64), (203, 29), (216, 27), (253, 23)]


def _source(K: int, J: int) -> str:
    return "\n".join([device_header(), tc_header(), f"""
struct Fill {{ __device__ void operator()(const i64* it, double* W) const {{
  for (int e = threadIdx.x; e < {K * J}; e += 128) W[e] = lcm_wp<const double>(it, 3)[e]; }} }};
extern "C" __global__ void __launch_bounds__(128) edge(const i64* items, const int* prefix, int n_items, int n_tiles) {{
  lcm_tc_expect<{K}, {J}>(items, prefix, n_items, n_tiles, 9, -1, Fill{{}});
}}"""])


@pytest.mark.skipif(not NVRTC.exists(), reason="NVRTC not installed")
@pytest.mark.parametrize("K,J", EDGES)
def test_edges_compile(K, J):
    rc, log = nvrtc_compile(_source(K, J))
    assert rc == 0, log[:2000]


@pytest.mark.gpu
@pytest.mark.parametrize("K,J", EDGES)
def test_edge_tables(K, J):
    import torch

    from pylcm_b200.runtime import get_context

    rng = np.random.default_rng(K)
    cols = 300  # three tiles, the last ragged
    W = np.where(rng.random((K, J)) < 0.3, 0.0, rng.random((K, J)))
    W[K // 2] = 0.0
    V = rng.normal(size=(J, cols))
    V[rng.random(V.shape) < 0.01] = -np.inf
    V[J - 1, 5], V[0, 7] = np.nan, np.inf
    dV, dW = torch.from_numpy(V).cuda(), torch.from_numpy(W).cuda()
    out = torch.full((K, cols), -7.0, dtype=torch.float32, device="cuda")
    items = torch.tensor([dV.data_ptr(), 0, out.data_ptr(), dW.data_ptr(), 0, 0, cols, cols, 0], dtype=torch.int64, device="cuda")
    prefix = torch.tensor([0, 3], dtype=torch.int32, device="cuda")
    mod = get_context(0).compile(_source(K, J), f"edge_{K}_{J}")
    mod.prepared("expect_tc", "edge", items.data_ptr(), prefix.data_ptr(), 1, 3, 128,
                 RegimeKernels.tc_shape(K, J)["smem"], grid=3)(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert mod.status() == 0
    got, want = out.cpu().numpy().astype(np.float64), _sum(W, V)
    fin = np.isfinite(V).all(axis=0)
    np.testing.assert_array_equal(got[:, ~fin], want[:, ~fin].astype(np.float32))
    assert (np.abs(got - want)[:, fin] <= 2e-6 * np.maximum(1.0, np.abs(want[:, fin]))).all()
