"""The chunks of the host entries when the caller leaves them open (CPU: the
choice is host arithmetic): never more than 8,192 columns or one block, and as
few as that allows where the arrays are pageable and their copies overlap
nothing."""
import pytest

from openifs_b200 import cloudsc


@pytest.mark.parametrize("nproma", [1, 24, 32, 128, 160, 3000, 8192, 8193, 20000])
@pytest.mark.parametrize("ngpblks", [1, 5, 16, 64, 256, 2048])
def test_chunks(built, nproma, ngpblks):
    most = max(1, 8192 // nproma)
    for klev, real in ((137, 8), (91, 8), (137, 4), (300, 8)):
        few = cloudsc.host_chunk_blocks(nproma, klev, ngpblks, real, page_locked=False)
        locked = cloudsc.host_chunk_blocks(nproma, klev, ngpblks, real, page_locked=True)
        for cb in (few, locked):
            assert 1 <= cb <= min(most, ngpblks)
        assert -(-ngpblks // few) == -(-ngpblks // most)
        assert locked <= few


def test_errors(built):
    for bad in ((0, 137, 4, 8), (32, 1, 4, 8), (32, 137, 0, 8), (32, 137, 4, 2)):
        with pytest.raises(cloudsc.CloudscError) as e:
            cloudsc.host_chunk_blocks(*bad)
        assert e.value.code == -2
