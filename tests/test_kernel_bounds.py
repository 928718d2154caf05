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


@pytest.mark.parametrize("gave_up", [False, True])
def test_shell_bounds_after_a_sort_that_gave_up(tmp_path, gave_up):
    """k_shell_bounds reads bin numbers from the sort's output.  When the sort gave up
    (ERR_SORT) some of that output was never written: no bounds then, and no store."""
    out = K.run(tmp_path, K.constants("ERR_SORT") + K.kernel_text("asg_shell", "k_shell_bounds") + f"""
int main()
{{
    std::vector<uint32_t> keys = {{0, 0, 3, 3, 3, 13, 26}}, start(27, 0u), end(27, 0u);
    int err = {int(gave_up)} ? ERR_SORT : 0;
    if (err) keys = {{0, 0, 0xcdcdcdcd, 3, 28, 0x7fffffff, 26}};
    run(1, 32, [&] {{ k_shell_bounds(keys.data(), (int)keys.size(), start.data(), end.data(), &err); }});
    for (int b : {{0, 3, 13, 26}}) std::printf("%u %u ", start[b], end[b]);
}}""")
    assert out.split() == (["0"] * 8 if gave_up else "0 2 2 5 5 6 6 7".split())


@pytest.mark.parametrize("pairs", [7, 2 ** 31 - 1, 2 ** 31, 2 ** 33])
def test_entries_of_more_pairs_than_numbers(tmp_path, pairs):
    """k_sorted_entries numbers the pairs in 32 bits.  A captured call whose pairs
    outgrew these has no pairs and reports ERR_CAP."""
    out = K.run(tmp_path, K.constants("ERR_SORT", "ERR_CAP") + K.kernel_text("asg_deposit", "k_sorted_entries") + f"""
int main()
{{
    const int order[] = {{2, 0, 1}};
    const uint2 entry[] = {{{{5, 0x7}}, {{6, 0xffffffff}}, {{9, 0x80000001}}}};
    const unsigned long long pairs = {pairs}ull;
    std::vector<uint2> list(3);
    std::vector<uint32_t> first(4, 77u);
    int err = 0;
    run(1, 32, [&] {{ k_sorted_entries(order, entry, 3u, &pairs, list.data(), first.data(), &err); }});
    for (uint32_t f : first) std::printf("%u ", f);
    std::printf("%d %d", list[0].x, err == ERR_CAP);
}}""")
    assert out.split() == ("2 3 32 0 9 0" if pairs < 2 ** 31 else "0 0 0 0 0 1").split()
