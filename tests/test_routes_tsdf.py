"""Where a ray cast steps over empty bricks (no GPU needed): marking them reads
the whole volume, so many rays and not too large a volume."""
import pytest


@pytest.mark.parametrize("dims,rays,want", [((256, 256, 256), (640, 480), 1), ((512, 512, 512), (640, 480), 1),
                                            ((1024, 1024, 1024), (640, 480), 0), ((1024, 1024, 1024), (200, 150), 0),
                                            ((1024, 1024, 1024), (1920, 1080), 1), ((768, 768, 768), (320, 240), 0),
                                            ((256, 256, 256), (320, 240), 0), ((512, 512, 64), (320, 240), 1),
                                            ((512, 512, 512), (320, 240), 1), ((48, 48, 48), (1280, 960), 0),
                                            ((4096, 4096, 4096), (4096, 4096), 1), ((4096, 4096, 4096), (64, 48), 0),
                                            ((2, 2, 2), (1, 1), 0)])
def test_bricks(dims, rays, want):
    from cvt_gb300 import _lib
    assert _lib.lib().cvtpm_tool_tsdf_bricks(*dims, *rays) == want
