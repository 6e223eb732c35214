"""GPU: the Q6_K GEMV adds the super-blocks of a row in their own order, whichever warp has them."""
import numpy as np
import pytest

from mtlqwen_b200 import device as D

pytestmark = pytest.mark.gpu


def ones(n, k):
  """Blocks of weights that are all 1: q = 33, scales and d 1."""
  block = np.zeros(210, np.uint8)
  block[:128], block[128:192], block[192:208], block[208:210] = 0x11, 0xaa, 1, np.frombuffer(np.float16(1).tobytes(), np.uint8)
  return np.tile(block, n * k // 256)


@pytest.mark.parametrize("m", [1, 8])
@pytest.mark.parametrize("k", [2048, 4096])  # one slab of eight super-blocks, two
def test_super_blocks_are_added_in_order(dev, k, m):
  n, rng = 32, np.random.default_rng(k + m)
  # one value of 11 bits in every super-block, of magnitudes so far apart that every order of the sum rounds differently
  sums = (rng.integers(1025, 2048, (m, k // 256)) * 2.0 ** rng.integers(0, 18, (m, k // 256)) * rng.choice([-1.0, 1.0], (m, k // 256))).astype(np.float32)
  x = np.zeros((m, k // 256, 256), np.float32)
  x[:, np.arange(k // 256), rng.integers(0, 256, k // 256)] = sums
  y = dev.empty((m, n))
  dev.linear(D.Q6_K, dev.array(ones(n, k)), n, k, dev.array(x.reshape(m, k)), m, y)
  dev.commit()
  chains = np.zeros((2, m), np.float32)  # super-blocks of even and of odd number
  for block in range(0, k // 256, 2):
    chains[0] += sums[:, block]
    chains[1] += sums[:, block + 1]
  assert y.download().tobytes() == np.repeat((chains[0] + chains[1])[:, None], n, axis=1).tobytes()
