"""Steps whose kernels come while their predecessors drain give, bit for bit, what launches in plain stream order give: every design
with its mixers and experts, prompts and single tokens, and latents so small that a block of the attention over them shares an SM
with blocks of the products behind it (both take tensor memory)."""

import pytest
import torch

from clockwork_b200 import ops
from clockwork_b200.cli import shape_config
from clockwork_b200.engine.step import StepEntry
from clockwork_b200.engine.trace import TraceSession
from clockwork_b200.weights import write_random_model
from tests.rapitar_configs import _dense, _latent, _mamba, _model, _moe, _wkv

pytestmark = pytest.mark.gpu

SMALL_LATENTS = _model(256, 128, 1e-5, [
    (_latent(4, 32, 16, 32, 48, 64, 1000.0, 0.2), _moe(8, 2, 64)),      # 64 columns: 50 KB of shared memory
    (_latent(4, 32, 16, 32, 112, 64, 1000.0, 0.2), _moe(16, 4, 128)),   # 128 columns: 98 KB
    (_latent(16, 64, 64, 64, 64, 128, 1000.0, 0.2), _dense(512)),
    (_mamba(4, 32, 32, 2, 4, 2), _moe(8, 2, 64)),
    (_wkv(4, 32), _moe(8, 2, 64)),
])
NAMES = ["rapitar-tiny", "gamesun-tiny", "kapolorn-tiny", "nuzulorn-tiny", "relerax-tiny", "dezolorn-tiny", "small-latents"]


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
@pytest.mark.parametrize("name", NAMES)
def test_overlapped_steps_have_the_bits_of_serial_ones(tmp_path, name, dtype):
    raw = SMALL_LATENTS if name == "small-latents" else shape_config(name)
    session = TraceSession(write_random_model(tmp_path, raw, seed=5), dtype, 1024, 16, graphs=False)
    tokens = [(7 * i * i + 3 * i) % raw["vocab"] for i in range(400)]

    def run():
        for rid in "ab":
            session.cache.open(rid)
        outs = [session.runner.step([StepEntry("a", tokens[:300], [0, 150, 299]), StepEntry("b", tokens[50:67], [16])])]
        for i in range(3):  # single tokens, then a portion beside one
            outs.append(session.runner.step([StepEntry("a", tokens[300 + i : 301 + i], [0]), StepEntry("b", tokens[67 + i : 68 + i], [0])]))
        outs.append(session.runner.step([StepEntry("a", tokens[303:380], [0, 76]), StepEntry("b", tokens[70:71], [0])]))
        outs = [o.clone() for o in outs]
        for rid in "ab":
            session.cache.close(rid)
        return outs

    try:
        ops.set_pdl(False)
        serial = run()
    finally:
        ops.set_pdl(True)
    differing = [i for i in range(15) if not all(torch.equal(a, b) for a, b in zip(run(), serial))]
    session.runner.check_status()
    assert all(torch.isfinite(o).all() for o in serial)
    assert not differing, f"runs {differing} of 15 differ from the run without overlap"
