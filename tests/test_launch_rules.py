"""Host-side rules that pick a kernel's form, asked on the CPU through tests/cpp/launch_rules.cc."""
INT_MAX = 2 ** 31 - 1


def test_rows_past_the_last_tile_do_not_wrap(launch_rules):
    """In tiles of several pieces a row index runs up to five pieces past M before it is compared with it."""
    rows = [INT_MAX - d for d in (0, 1, 127, 128, 511, 512, 639, 640, 641, 100000)]
    for m, (pieces,) in zip(rows, launch_rules([("pieces", m, 64, 148) for m in rows])):
        last_tile = (m - 1) // (128 * pieces) * (128 * pieces)
        assert pieces == 1 or last_tile + 127 + 128 * pieces <= INT_MAX, m
    assert launch_rules([("pieces", INT_MAX - 640, 64, 148)]) == [(4,)]


def test_pieces_by_rows(launch_rules):
    """Two tiles or more for each of four teams of every SM, and K up to 256."""
    one, two, four = 8 * 128 * 148, 2 * 8 * 128 * 148, 4 * 8 * 128 * 148
    rows = {1: 1, one: 1, two - 1: 1, two: 2, four - 1: 3, four: 4, 2 * four: 4}
    assert launch_rules([("pieces", m, 256, 148) for m in rows]) == [(p,) for p in rows.values()]
    assert launch_rules([("pieces", four, 272, 148), ("pieces", four // 2, 16, 74)]) == [(1,), (4,)]


def test_column_blocks_follow_the_tiles_of_a_convolution(launch_rules):
    """Tiles of 32 to 64 columns: blocks of 16 where all warps share a CTA's only tile, the widest where a team takes it.  Sizes around
    a wave of 148 tiles, where ceil(M / 128) and the spatial tiles differ."""
    sizes = [(n, hw, k, stride, oc) for hw, k, stride, images in ((56, 3, 1, (4, 5, 6, 7)), (19, 3, 1, (44, 45, 46, 52, 53)), (33, 3, 1, (16, 17, 18)),
                                                                  (7, 3, 1, (384, 385, 386, 387)), (75, 3, 1, (2, 3, 4)), (38, 3, 2, (46, 50)), (112, 1, 2, (5, 6)))
             for n in images for oc in (32, 64)]
    one = {}
    for (n, hw, k, stride, oc), (m_tiles, n_tiles, data, blk_w, one_each) in zip(sizes, launch_rules([("conv", n, hw, hw, k, stride, 64, oc) for n, hw, k, stride, oc in sizes])):
        out = (hw + stride - 1) // stride
        assert m_tiles >= -(-n * out * out // 128)
        assert one_each == (m_tiles * n_tiles <= 148 // n_tiles * n_tiles)
        assert blk_w == (16 if one_each and data >= 32 else data), (n, hw, oc)
        one[n, hw, oc] = one_each
    # 147 tiles by pixels, but 168 and more by 8 x 16 pieces of the images
    assert [one[n, 56, 64] for n in (4, 5, 6, 7)] == [1, 1, 0, 0] and not one[47 - 1, 19, 64] and not one[17, 33, 64] and not one[385, 7, 64] and not one[3, 75, 64]


def test_output_rows_of_an_im2col_block_follow_the_device(launch_rules):
    """Several rows only where six blocks are left for every SM of the device there is."""
    lenet, stem = (28, 28, 1, 5, 5, 1, 1, 0), (230, 230, 3, 7, 7, 2, 2, 0)
    sizes = [(n, layer, sms) for layer in (lenet, stem) for n in (1, 13, 64, 1000) for sms in (74, 148, 296)]
    rows = {}
    for (n, layer, sms), (out_rows, blocks, _) in zip(sizes, launch_rules([("im2col", n) + layer + (sms,) for n, layer, sms in sizes])):
        assert out_rows >= 1 and (out_rows == 1 or blocks >= 6 * sms), (n, layer, sms)
        rows[n, layer, sms] = out_rows
    assert [rows[64, lenet, sms] for sms in (74, 148, 296)] == [3, 1, 1]
    assert rows[1000, lenet, 148] > 8 and rows[1, lenet, 74] == 1 and rows[64, stem, 148] == 2
