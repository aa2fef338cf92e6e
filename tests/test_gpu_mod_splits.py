"""The modular products' bits do not depend on the split of K, which
follows the number of tiles: a lone product against the same one inside a
batch, on sums that cancel and outputs near the accuracy check's line."""
import pytest
import torch

from test_gpu_mod import _gemm

pytestmark = pytest.mark.gpu


def _lone_and_batched(lib, A, B, reps=16):
    """A @ B alone, and (the same rows) among reps * M rows and as reps
    replicas of both: fewer K slices in each."""
    M, N = A.shape[0], B.shape[1]
    lone = _gemm(lib, 1, A, B, torch.zeros(M, N, dtype=torch.float64, device="cuda"))
    C = torch.zeros(reps, M, N, dtype=torch.float64, device="cuda")
    rows = _gemm(lib, 1, A.expand(reps, *A.shape).contiguous(), B.unsqueeze(0).expand(reps, *B.shape), C)
    both = _gemm(lib, 1, A.expand(reps, *A.shape).contiguous(), B.expand(reps, *B.shape).contiguous(), C)
    for r in range(reps):
        assert torch.equal(rows[r], lone) and torch.equal(both[r], lone), r
    return lone


@pytest.mark.parametrize("depth", [None, 27, 33, 40, 50])
@pytest.mark.parametrize("M,N,K", [(250, 300, 8192), (100, 100, 40000)])
def test_cancelling_sums(gpulib, M, N, K, depth):
    """Sums of about 2^-depth of their terms; exactly 0 without one."""
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn(M, K // 2, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(K // 2, N, generator=g, device="cuda", dtype=torch.float64)
    r = torch.rand(K // 2, N, generator=g, device="cuda", dtype=torch.float64)
    B2 = B if depth is None else B * (1.0 + 2.0 ** -depth * r)
    out = _lone_and_batched(gpulib, torch.cat([A, A], 1), torch.cat([B, -B2], 0))
    if depth is None:
        assert bool((out == 0.0).all())


@pytest.mark.parametrize("M,N,K", [(250, 300, 8192)])
def test_outputs_at_the_check(gpulib, M, N, K):
    """Rows whose large elements meet the columns' small ones, by factors on
    both sides of the line below which an output is recomputed."""
    g = torch.Generator(device="cuda").manual_seed(9)
    A = torch.randn(M, K, generator=g, device="cuda", dtype=torch.float64)
    B = torch.randn(K, N, generator=g, device="cuda", dtype=torch.float64)
    A[:, ::2] *= 2.0 ** -(4.0 + 8.0 * torch.rand(M, 1, generator=g, device="cuda", dtype=torch.float64))
    B[1::2] *= 2.0 ** -(4.0 + 8.0 * torch.rand(1, N, generator=g, device="cuda", dtype=torch.float64))
    _lone_and_batched(gpulib, A, B)


@pytest.mark.parametrize("precision", ["fp64", "df64"])
def test_replicas_are_their_lone_solves(gpulib, precision):
    """Twelve replicas at a size whose products are split differently alone."""
    from fricc_gb300.batch import mp2_device
    from fricc_gb300.friccsd import FRICCSDGPU
    from fricc_gb300.rccsd_dense import DeviceERIs
    from fricc_gb300.replicas import FusedReplicaBatch
    from fricc_gb300.rng import GlibcRand
    from fricc_gb300.synthetic import DeviceSystem
    E = DeviceERIs.from_system(DeviceSystem(17, 83, 800, 0.04, seed=5))
    m, seeds = 150_000, list(range(40, 52))
    fb = FusedReplicaBatch(E, {"m_keep": m}, seeds, precision=precision)
    for _ in range(2):
        fb.step()
    settings = {"compression": "fri", "sampling_method": "systematic", "verbose": False, "m_keep": m,
                "compressed_contractions": ["O^2V^4", "O^3V^3", "O^4V^2"]}
    for r in (0, 5, 11):
        lone = FRICCSDGPU(E, settings, rn_draw=GlibcRand(seeds[r]), precision=precision)
        t1, t2 = mp2_device(E)
        for _ in range(2):
            t1, t2 = lone.update_amps(t1, t2)
        assert torch.equal(t1, fb.t1[r]) and torch.equal(t2, fb.t2[r]), r
