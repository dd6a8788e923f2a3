"""Single tokens of retention with the state's packs in shared memory: up to 4, 8 and 16 packs a thread (the last one's 64 KB), one pack less and a row
of threads that has none, held as the step of the other sizes is."""
import pytest
import torch

import test_chunk_scans_gpu as scans

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,V,rot", [(2, 64, 128, 64), (2, 128, 64, 32), (1, 128, 128, 128), (1, 127, 128, 0), (3, 65, 64, 2), (1, 40, 100, 8)])
def test_packs_of_a_thread(N, K, V, rot):
    scans.test_one_token_of_every_request_in_one_retention_kernel(torch.float32, N, K, V, rot)
