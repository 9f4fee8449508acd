"""The bit budget of a layer without tensor arithmetic."""
import random

import torch

from actnn_b200.qscheme import target_bits


def test_the_product_is_the_one_torch_gives():
    rng = random.Random(3)
    for i in range(5000):
        n = rng.randint(1, 5000)
        average = torch.tensor(rng.randint(n, 8 * n)).float() / n          # what the joint allocation leaves
        for bits in (average, torch.tensor(rng.uniform(0.5, 9.0)), torch.tensor(rng.randint(1, 8), dtype=torch.int32), 2, 3.7):
            assert target_bits(bits, n) == int(bits * n)
