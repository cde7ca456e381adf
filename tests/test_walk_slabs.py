"""The walk's slab test (traverse.cuh visit_slots) takes its plane bytes from a byte dot product into the bits of 65536
and takes 65536 off again: restated here, every byte must come out as itself, so that the test is fma(q, a, o) bit for
bit."""
import numpy as np

F32 = np.float32


def test_plane_bytes_come_out_exactly():
    q = np.arange(256, dtype=np.uint32)
    for c in range(4):
        other = np.uint32(0xA5C3F017) & ~np.uint32(0xFF << (8 * c))
        word = other | (q << np.uint32(8 * c))
        weight = 128 << (8 * c)  # one byte of the dot product's second operand
        dot = sum(((word >> np.uint32(8 * k)) & 0xFF) * np.uint32((weight >> (8 * k)) & 0xFF) for k in range(4))
        raised = (np.uint32(0x47800000) + dot.astype(np.uint32)).view(F32)
        assert np.array_equal(raised, (65536 + q).astype(F32))
        assert np.array_equal(raised + F32(-65536), q.astype(F32))
