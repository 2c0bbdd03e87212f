"""Which prompt portions have their attention's work cut along the keys (on the host)."""
import pytest

from spite_b200.cache import Window
from spite_b200.kernels.cuda import attention_cut_pays

BLOCKS, KEY_BYTES = 148, 512                                  # keys and values of 128 bfloat16


# 40 heads, 8 kv heads (25 tokens a row tile): (first position, tokens) of the portions and which form was faster
@pytest.mark.parametrize("segments,cut", [
    ([(6144, 2048)], True), ([(7192, 1000)], True), ([(7692, 500)], True), ([(8092, 100)], True), ([(8142, 50)], True), ([(7500, 683)] * 3, True),
    ([(0, 2048)], False), ([(1000, 1048)], False), ([(500, 500)], False), ([], False)])
@pytest.mark.parametrize("window", [Window("full", 0), Window("chunk", 8192)], ids=["full", "chunk"])
def test_the_faster_form(segments, cut, window):
    assert attention_cut_pays(tuple(segments), window, 50, 8, BLOCKS, KEY_BYTES) is cut


@pytest.mark.parametrize("segments,heads,key_bytes,cut", [
    ([(122880, 8192)], (50, 8), 512, False), ([(57344, 8192)], (50, 8), 512, False), ([(24576, 8192)], (50, 8), 512, False), ([(129024, 2048)], (50, 8), 512, True),
    ([(63488, 2048)] * 4, (50, 8), 512, False), ([(30720, 2048)] * 4, (50, 8), 512, False), ([(122880, 8192)], (64, 8), 512, False),
    ([(126976, 4096)], (256, 16), 512, False), ([(28672, 4096)], (256, 16), 512, True), ([(130072, 1000)], (256, 16), 512, True),
    ([(122880, 8192)], (32, 4), 256, True), ([(57344, 8192)], (32, 4), 256, True)])
def test_keys_beyond_the_cache(segments, heads, key_bytes, cut):
    """Long contexts, measured on both forms: what whole items share in L2 outweighs even shares, unless many blocks would have none."""
    assert attention_cut_pays(tuple(segments), Window("full", 0), *heads, BLOCKS, key_bytes) is cut


def test_a_window_bounds_what_a_cut_can_give():
    """128 keys a token are three tiles: no item is long enough to share."""
    assert attention_cut_pays(((8092, 100),), Window("full", 0), 50, 8, BLOCKS, KEY_BYTES)
    assert not attention_cut_pays(((8092, 100),), Window("sliding", 128), 50, 8, BLOCKS, KEY_BYTES)


@pytest.mark.parametrize("segments", [[(0, 1)], [(0, 33), (4000, 900), (7, 129)], [(100, 2048)] * 30, [(131000, 2048)], [(0, 16400)]])
@pytest.mark.parametrize("window", [Window("full", 0), Window("chunk", 512), Window("sliding", 1000)], ids=["full", "chunk", "sliding"])
@pytest.mark.parametrize("pair,heads", [(50, 8), (16, 1), (256, 1), (256, 40)])
def test_against_every_item_dealt_out(segments, window, pair, heads):
    """The estimate takes five of the blocks and draws a line through the items of a portion; dealing every item out to every block gives the
    same answer unless the two forms lie within a fifth of one another."""
    items = []
    for start, n in reversed(segments):
        for t in reversed(range(0, n, pair)):
            last = start + min(n, t + pair) - 1
            items += [6 + (last - window.lowest_visible(start + t)) / 64 + 1] * heads
    sums = [0.0] * BLOCKS
    for i, cost in enumerate(items):
        round_, at = divmod(i, BLOCKS)
        sums[BLOCKS - 1 - at if round_ & 1 else at] += cost
    seen = sum(s + n - window.lowest_visible(s) for s, n in segments) * heads * KEY_BYTES
    whole, cut = max(sums), max(8.0, sum(items) / BLOCKS) * (1 + 0.17 * max(0.0, 1 - 1e8 / max(seen, 1))) + 24
    if not 0.8 < whole / cut < 1.25:
        assert attention_cut_pays(tuple(segments), window, pair, heads, BLOCKS, KEY_BYTES) is (cut < whole)


def test_the_layers_of_a_step_ask_once():
    """48 layers, three of four with another window: two answers are made, and other portions make others."""
    segments = tuple((100 + i, 40 + i) for i in range(64))
    attention_cut_pays.cache_clear()
    for layer in range(48):
        attention_cut_pays(tuple(segments), Window("chunk", 8192) if layer % 4 else Window("full", 0), 50, 8, BLOCKS, KEY_BYTES)
    assert attention_cut_pays.cache_info().misses == 2
    attention_cut_pays(segments[:-1] + ((163, 104),), Window("full", 0), 50, 8, BLOCKS, KEY_BYTES)
    assert attention_cut_pays.cache_info().misses == 3
