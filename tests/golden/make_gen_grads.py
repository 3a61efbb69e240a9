"""Writes gen_grads.json: digests of the generator's gradients over four training steps.

The digests were written by the first form of the gradient kernels (one launch per layer and sum),
whose order of additions every later form keeps. Runs on the GPU, from the repository's root:
python tests/golden/make_gen_grads.py [output]"""
import hashlib
import json
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
# edge, batch, tensor-core mode
CASES = [(128, 16, 1), (128, 3, 1), (128, 2, 0), (128, 2, 3), (64, 16, 1), (64, 5, 1), (64, 3, 0), (48, 5, 1), (32, 16, 1),
         (32, 1, 1), (16, 4, 1), (96, 2, 1), (192, 1, 1)]
STEPS = 4


def digests(edge, batch, mode):
    """SHA-256 of the gradients after each of four steps on snapshots of swept chains."""
    from nanomagmc_gb300.warmstart import Generator, heisenberg_sampler

    rng = np.random.default_rng(edge + batch)
    T, B = rng.uniform(0.3, 1.5, batch), rng.uniform(0.0, 1.0, batch)
    s = heisenberg_sampler(edge, 0.5, T, B, seed=5)
    gen = Generator(edge, capacity=batch, seed=6)
    gen.tensor_cores(mode)
    s.sweep(10)
    gen.add_snapshots(s, np.arange(batch), np.stack([T, B, np.full(batch, 0.5)], 1))
    s.close()
    out = []
    for step in range(STEPS):
        gen.train_step(np.arange(batch), np.clip(rng.uniform(0.0, 1.0, batch), 0.05, 1.0), 1e-3)
        out.append(hashlib.sha256(np.ascontiguousarray(gen.grads(), np.float32).tobytes()).hexdigest())
    return out


if __name__ == "__main__":
    sys.path.insert(0, os.environ.get("TREE", ROOT))
    out = {"%d_%d_%d" % c: digests(*c) for c in CASES}
    with open(sys.argv[1] if len(sys.argv) > 1 else os.path.join(os.path.dirname(os.path.abspath(__file__)), "gen_grads.json"), "w") as f:
        json.dump(out, f, indent=1)
