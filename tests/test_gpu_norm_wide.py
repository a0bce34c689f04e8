"""Norms of rows of whole packets where the kernel that takes them changes: wide rows backward and forward, bf16 rows of few
packets forward, fp32 rows while they are few.  Row lengths and counts on both sides of the limits, against the oracle."""
import pytest

import test_gpu_norm_teams as T

pytestmark = pytest.mark.gpu

# rows that one warp still holds and the first ones beyond; 16 warps with two, three and four packets a thread; too long
FP32 = [(1999, 2048), (2000, 2048), (300, 1792), (70, 2052), (65, 3072), (1500, 3008), (1500, 3012), (100, 4096), (66, 4100),
        (130, 6144), (130, 6148), (300, 8192), (66, 8196), (3, 5120), (888, 512), (889, 512), (444, 1280), (445, 1280)]
# the pair kernel's last rows and the next; one packet per thread and two; the forward's limits by length and by elements
BF16 = [(300, 1536), (300, 1544), (3, 1544), (130, 4096), (130, 4104), (66, 8192), (66, 8200), (2075, 4096), (700, 8), (4000, 256),
        (5000, 248), (8854, 960), (8855, 960), (300, 1600)]


@pytest.mark.parametrize("n,c", FP32)
def test_layernorm(n, c):
    T.test_layernorm_teams_vs_oracle(n, c)


@pytest.mark.parametrize("n,c", FP32)
def test_rmsnorm(n, c):
    T.test_rmsnorm_teams_vs_oracle(n, c, "f32")


@pytest.mark.parametrize("n,c", BF16)
def test_rmsnorm_bf16(n, c):
    T.test_rmsnorm_teams_vs_oracle(n, c, "bf16")
