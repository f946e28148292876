"""The bytes model of the bench follows the words that a handle has, not its
size: FP32 domains that kept whole words move 224 bytes a node."""
import bench


def test_bytes_follow_the_handles_words():
    assert bench.bytes_per_node("fp32", dict(blocks=100, short_blocks=0)) == 224
    assert bench.bytes_per_node("fp32", dict(blocks=100, short_blocks=100)) == 188
    assert bench.bytes_per_node("fp32", dict(blocks=100, short_blocks=50)) == 206
    assert bench.bytes_per_node("fp64", dict(blocks=100, short_blocks=0)) == 376
    assert bench.bytes_per_node("fp32", dict(blocks=0, short_blocks=0)) == 224
