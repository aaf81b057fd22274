"""Launches are shaped for the device they run on, not for the first one used."""
from host_runtime import i64, library, log


def test_teams_follow_the_current_device():
    h = library()
    h.fake_log()
    seen = []
    try:
        for device, sms in ((0, 148), (40, 60), (0, 148), (41, 148)):
            h.fake_device(device, sms)
            h.h_fp12_mul(*i64(1000))  # two values to a scheduler: 1,184 of 148 SMs, 480 of 60
            (launch,) = log(h)[0]
            seen.append("Twelve" in launch[0])
    finally:
        h.fake_device(0, 148)
    assert seen == [True, False, True, True]
