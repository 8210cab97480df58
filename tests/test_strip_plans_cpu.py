"""Strip plans are kept: three handles' worth of them (48) asked for in turn are
searched for once."""
import ctypes


def test_plans_in_turn_are_searched_once(built_lib):
    u = ctypes.c_uint
    whole, n, p = u(), (u * 3)(), (u * 3)()
    keys = [(bands, cols, kk, 152) for bands in range(160, 480, 20) for cols, kk in ((320, 4), (640, 4), (640, 1))]
    assert len(keys) == 48
    count = ctypes.c_ulonglong()

    def ask():
        plans = []
        for bands, cols, kk, ctas in keys:
            assert built_lib.pdflow_strip_units(bands, cols, kk, ctas, ctypes.byref(whole), n, p) == 0
            plans.append((whole.value, tuple(n), tuple(p)))
        assert built_lib.pdflow_strip_plan_count(ctypes.byref(count)) == 0
        return plans, count.value

    first, searched = ask()
    again, then = ask()
    assert again == first and then == searched
