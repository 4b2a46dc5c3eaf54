"""Sizes at which a query or a camera takes a given route through the traversal, for the tests
that are about that route; test_routes_cpu.py holds them against the library's own choice."""


def warps(sms: int) -> int:
    """Resident warps of the one-kernel route, by which the library chooses."""
    return 32 * sms


def two_pass_rays(sms: int, node_format: int, leaf_size: int) -> int:
    """Rays of one scene that run as a regular and a deferred pass (a ragged last batch)."""
    per_warp = 420 if node_format == 0 and leaf_size == 1 else 130
    return per_warp * warps(sms) + 45


def packet_image(sms: int, n_tris: int):
    """Width and height of a camera whose batches start with a packet descent."""
    width = 1021
    pixels = max(120 * warps(sms) + 1, 640 * n_tris)
    return width, -(-pixels // width)
