"""Where the single-pass attention backward splits its last round of key tiles over the SMs (host arithmetic; needs no GPU)."""
import pytest


@pytest.mark.parametrize("B,S,H,Hkv,split", [
    (1, 128, 8, 4, False), (2, 128, 8, 2, False), (48, 128, 8, 8, False),           # items of one tile: a few units, no pair to split
    (37, 128, 8, 4, False), (148, 256, 4, 1, False),                               # whole rounds
    (16, 256, 8, 4, False), (12, 512, 8, 4, False), (32, 512, 8, 8, False), (17, 1024, 8, 4, False), (64, 1024, 8, 4, False),   # saves less than it costs
    (1, 512, 8, 4, True), (3, 1920, 8, 4, True), (8, 2048, 8, 4, True), (48, 2048, 8, 4, True), (1, 8192, 8, 2, True)])
def test_a_round_is_split_only_where_that_saves_more_than_the_merge_costs(B, S, H, Hkv, split):
    from parameter_golf_b200.ops import native
    C = native.load_raw()
    need = C.attn_bwd_part_floats(B, S, H, Hkv)
    assert need == (C.attn_bwd_part_floats() if split else 0)
