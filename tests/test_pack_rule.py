"""When BatchPipeline packs fields: sizes where both ways were timed (no GPU)."""
import pytest


@pytest.mark.parametrize("frames,D,rate,C,rays,S,want", [
    (1, 64, 8, 16, 256, 32, (False, False, False)), (1, 64, 8, 16, 4096, 96, (False, True, True)),
    (1, 64, 8, 16, 16384, 96, (True, True, True)), (1, 64, 8, 3, 16384, 96, (True, True, True)),
    (1, 128, 8, 16, 4096, 32, (False, False, False)), (1, 128, 8, 16, 131072, 32, (True, True, True)),
    (1, 256, 8, 16, 16384, 32, (False, False, False)), (1, 256, 8, 16, 131072, 96, (True, True, True)),
    (1, 256, 8, 16, 1 << 20, 96, (True, True, True)),
    (4, 256, 8, 16, 256, 32, (False, False, False)), (4, 256, 8, 16, 16384, 96, (False, False, False)),
    (4, 256, 8, 16, 131072, 32, (False, False, True)), (4, 256, 8, 3, 131072, 96, (False, True, True)),
    (4, 256, 8, 16, 1 << 22, 64, (True, True, True)), (8, 128, 8, 16, 4096, 96, (False, False, False)),
    (1, 512, 8, 16, 131072, 32, (False, False, True)), (1, 256, 4, 16, 131072, 96, (True, True, True))])
def test_rule(frames, D, rate, C, rays, S, want):
    from sailor_gb300.batch import pack_pays
    assert pack_pays(rays * S, frames, D // rate, rate, C) == want
