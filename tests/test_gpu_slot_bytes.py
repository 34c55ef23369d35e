"""The bytes a server counts for a slot are the device memory it holds, the
step's scratch among them, so a byte budget is kept."""
import importlib

import pytest
import torch

from tests.helpers import pkg, planets

serving = importlib.import_module("web-exoplasim_b200.serving")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("truncation,levels,slots", [(21, 5, 1024), (42, 10, 128), (63, 10, 64)])
def test_slot_bytes_are_the_memory_an_engine_takes(truncation, levels, slots):
    pkg.Engine(truncation, levels, 1).close()  # the library's kernels are loaded
    before = torch.cuda.mem_get_info()[0]
    e = pkg.Engine(truncation, levels, slots)
    try:
        held = before - torch.cuda.mem_get_info()[0]
        # about ten allocations, each rounded up to 2 MiB; the scratch is above 100 MiB in each case
        assert abs(held - slots * e.slot_bytes()) <= 32 << 20, (held, slots * e.slot_bytes())
    finally:
        e.close()
    assert serving.slot_bytes(truncation, levels) == pytest.approx(held / slots, rel=0.01)


def test_server_refuses_a_block_one_percent_above_its_budget():
    e = pkg.Engine(42, 10, 1)
    need = e.slot_bytes()
    e.close()
    for share, status in ((0.99, "rejected"), (1.01, "finished")):
        server = pkg.NativeServer(budget_bytes=share * need, block_slots=1, chunk_steps=8, mode=1)
        try:
            run = server.submit(planets.make_planet(321, truncation=42, levels=10), 8)
            for _ in range(200):
                if server.pump() == 0:
                    break
            assert server.poll(run)[0] == status
        finally:
            server.close()
