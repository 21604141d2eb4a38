"""An attention layer's step in one C call: what a later launch would refuse or take for granted is refused ahead of the first one, which writes the caches."""
import pytest

from krasis_b200 import seqops as ops

# addresses that nothing may be read from: 16-byte aligned, and host memory for the layout alone
AT = {n: 0x1000000 * (i + 1) for i, n in enumerate(("proj", "positions", "seq_of", "pages", "kc", "vc", "fmha", "work", "out"))}


def _call(layout=((0, 130, 62, 3), (130, 1, 5, 1)), **kw):
    import numpy as np
    a = dict(AT, T=131, H=4, G=2, d=128, dv=128, max_pages=3, page_size=64, dt_cache=1, dt_out=1, scale=0.1, window=1 << 20, softcap=0.0, min_long=128, work_bytes=1 << 40, S=2)
    a.update(kw)
    table = np.array(layout, dtype=np.int32)
    rc = ops.load().kb2_seq_attention_step(a["proj"], 1024, table.ctypes.data, a["S"], a["T"], a["H"], a["G"], a["d"], a["dv"], None, None, None, 1e-6, None, 0,
                                           a["positions"], a["seq_of"], a["pages"], a["max_pages"], a["page_size"], a["kc"], a["vc"], a["dt_cache"], 0, 0, 1.0, 0,
                                           a["scale"], a["window"], a["softcap"], None, None, a["min_long"], 0, a["fmha"], a["work"], a["work_bytes"], a["out"],
                                           a["dt_out"], 0, None)
    return rc, ops.load().kb2_seq_last_error().decode()


@pytest.mark.parametrize("kw", [
    {"d": 64}, {"d": 256}, {"dv": 64}, {"dv": 192}, {"dt_cache": 0}, {"dt_out": 0}, {"fmha": None}, {"scale": 0.0}, {"scale": -1.0}, {"out": AT["out"] + 8},       # the tensor cores' portions
    {"page_size": 0}, {"page_size": -64}, {"max_pages": 0}, {"H": 0}, {"H": 5}, {"G": 0}, {"T": 0}, {"S": 0}, {"window": 0}, {"softcap": -1.0}, {"dt_cache": 2},
    {"kc": AT["kc"] + 8}, {"vc": AT["vc"] + 2}, {"min_long": 0, "dv": 513}, {"min_long": 0, "d": 2000}, {"work": AT["work"] + 4}, {"work_bytes": 1000},
    {"proj": None}, {"positions": None}, {"seq_of": None}, {"pages": None}, {"kc": None}, {"work": None}, {"out": None},
    {"T": 130}, {"T": 132}, {"layout": ((0, 130, 62, 3), (129, 1, 5, 1))}, {"layout": ((1, 130, 62, 3), (131, 1, 5, 1))}, {"layout": ((0, 132, 60, 3), (132, -1, 5, 1))},
    {"layout": ((0, 130, -1, 3), (130, 1, 5, 1))}, {"layout": ((0, 130, 2 ** 31 - 100, 3), (130, 1, 5, 1))}, {"layout": ((0, 130, 62, 4), (130, 1, 5, 1))},
])
def test_refused_ahead_of_the_first_launch(kw):
    rc, text = _call(**kw)
    assert rc == 2 and text.startswith("attention_step"), (rc, text)


def test_pages_that_do_not_hold_a_long_portion():
    rc, text = _call(layout=((0, 130, 63, 3), (130, 1, 5, 1)))            # 193 positions in three pages of 64
    assert rc == 4 and text.startswith("attention_step"), (rc, text)


@pytest.mark.parametrize("blocks", [1, 2, 3, 7, 20, 147, 148, 149, 296, 297, 5000])
@pytest.mark.parametrize("least", [8, 32])
def test_pieces_of_a_step_and_of_its_replay(blocks, least):
    """Cut by its own keys or by the room: the pieces that have keys are the same, and a row is joined in both or in neither."""
    pieces = ops.load().kb2_seq_key_pieces

    def cut(keys, n):
        size = -(-(-(-keys // n)) // least) * least
        return [(a, min(keys, a + size)) for a in range(0, keys, size)]
    for room in (1, 8, 40, 512, 4096, 1 << 20):
        for keys in sorted({1, 7, 31, 32, 33, 64, 65, 500, 2047, 2048, 2049, 4000, room} | {room - 1 if room > 1 else 1}):
            if keys <= room:
                one, many = pieces(blocks, keys, room, least), pieces(blocks, room, room, least)
                assert 1 <= one <= many <= 64 and (one == 1) == (many == 1) and cut(keys, one) == cut(keys, many)
                assert many == 1 or blocks * many <= 2 * 148


def test_workspace_of_nothing():
    assert ops.load().kb2_seq_attention_step_workspace(None, 2, 4, 2, 128, 128, 3, 64, 1 << 20, 128, 0) == 0


def test_one_layout():
    """The C interfaces see what StepTables.layout was set to, and it cannot be changed in place."""
    import ctypes
    tb = ops.StepTables([([5, 6, 7], 60, 0, [2, 1]), ([8], 9, 1, [0])], "cpu")

    def seen():
        return [tuple((ctypes.c_int * 4).from_address(tb.layout_ptr + 16 * i)) for i in range(tb.S)]
    assert seen() == [(0, 3, 60, 2), (3, 1, 9, 1)] and list(tb.layout) == [(0, 3, 60, [2, 1]), (3, 1, 9, [0])]
    tb.layout = [(0, 3, 30, [2]), (3, 1, 10, [0])]
    assert seen() == [(0, 3, 30, 1), (3, 1, 10, 1)]
    with pytest.raises(TypeError):
        tb.layout[0] = (0, 3, 0, [])
