"""CPU tests of kernels on the inputs of a call that is about to report an error:
what the kernels after them read must still be in range."""
import pytest

import cpu_kernel as K


@pytest.mark.parametrize("room", [1, 5, 9, 10, 12, 100])
def test_item_list_fills_every_item_that_runs(tmp_path, room):
    """k_item_list with more items than the arrays hold: every item below the room
    has its tile (the deposit runs these), and nothing beyond it is written."""
    out = K.run(tmp_path, K.constants("ERR_CAP", "MERGE_FEW") + K.kernel_text("asg_deposit", "k_item_list") + f"""
int main()
{{
    const uint32_t off[] = {{0, 1, 4, 5, 11, 12, 24, 25}};  // tiles of 1, 3, 1, 6, 1, 12 and 1 items
    const int T = 7;
    const uint32_t room = {room};
    std::vector<uint32_t> tile(room, 0xdeadbeefu), merge(T, 0u);
    std::vector<int> counters(8, 0);
    int err = 0;
    run(1, 32, [&] {{ k_item_list(off, T, room, tile.data(), merge.data(), counters.data(), &err); }});
    std::printf("%d\\n", err);
    for (uint32_t t : tile) std::printf("%d ", (int)t);
    std::printf("\\n%d %d\\n", counters[1], counters[4]);
}}""").split("\n")
    want = [0, 1, 1, 1, 2] + [3] * 6 + [4] + [5] * 12 + [6]
    got = [int(t) for t in out[1].split()]
    assert got[:len(want)] == want[:room]
    assert (int(out[0]) != 0) == (room < len(want))
    if room >= len(want):
        assert out[2] == "2 1"
