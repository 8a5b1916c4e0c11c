"""Which form of the attention kernel a call takes (attention_form, csrc/flash_attn.cu), on a device of 148 SMs: calls whose forms
were all timed, the taken one within a tenth of the fastest, and never a tenth behind what the call would run as without pairs of
CTAs.  No device is needed."""
import pytest

from fractaltensor_b200._lib import lib

FULL, CAUSAL = (0, -1, 0), (1, -1, 0)
TIMED = [  # (batch, head) entries, keys, mask; us as CTAs of 256 rows, halves, pairs; the form without pairs; the form taken
    (16, 256, FULL, (8.2, 7.2, 7.4), 2, 2), (7, 512, FULL, (13.0, 10.4, 9.5), 2, 2), (99, 512, FULL, (30.4, 34.3, 19.3), 1, 3),
    (40, 1024, FULL, (39.5, 40.1, 26.8), 1, 3), (16, 2048, FULL, (35.9, 43.0, 33.2), 1, 3), (20, 2048, FULL, (68, 63, 45), 2, 3),
    (4, 4096, FULL, (63, 37, 33), 2, 3), (256, 2048, FULL, (490, 574, 438), 1, 3),
    (15, 256, CAUSAL, (8.3, 6.9, 8.0), 2, 2), (66, 512, CAUSAL, (12.8, 19.7, 13.9), 1, 1), (36, 1024, CAUSAL, (20.4, 26.7, 17.4), 1, 3),
    (16, 2048, CAUSAL, (37, 28, 23.4), 2, 3), (84, 3328, CAUSAL, (266, 294, 225), 1, 3),
    (77, 768, (1, 64, 0), (24.1, 29.0, 28.7), 1, 1), (42, 3584, (1, 1306, 0), (110, 139, 111), 1, 3),
    (42, 1024, (1, 751, 392), (40, 39, 29.5), 1, 3),
    # at most two rounds of pairs of SMs: tiles that are nearly all equally long
    (12, 2304, (1, 161, 745), (25.9, 29.6, 31.3), 1, 1), (6, 4096, (1, 723, 1049), (38.3, 37.4, 41.5), 2, 2),
    (28, 1280, (1, 997, 542), (24.6, 31.7, 25.6), 1, 3),
]


@pytest.mark.parametrize("n_bh,S,mask,us,without,taken", TIMED)
def test_form_of_timed_calls(n_bh, S, mask, us, without, taken):
    form = lib.ftb_flash_attn_form(n_bh, S, *mask, 148)
    assert form == taken
    assert us[form - 1] <= 1.1 * min(us) and us[form - 1] <= 1.05 * us[without - 1]


def test_what_is_no_call():
    assert lib.ftb_flash_attn_form(0, 256, 0, -1, 0, 148) == lib.ftb_flash_attn_form(1, 255, 0, -1, 0, 148) == 0
    assert lib.ftb_flash_attn_form(1, 256, 1, -1, -1, 148) == 0
