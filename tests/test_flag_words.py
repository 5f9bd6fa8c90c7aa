"""Flag words that several CTAs report into are only ever ORed: a CTA that
stores or exchanges the word can take back what another one reported (a wait
that gave up at the last barrier, which the storing CTA passed).  Which of the
two comes last is a matter of time, so the source is what shows it."""

import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yggdrax_b200",
                    "csrc")


@pytest.mark.parametrize("path", sorted(glob.glob(os.path.join(CSRC, "*.cu*"))),
                         ids=os.path.basename)
def test_flag_words_are_only_ored(path):
    text = re.sub(r"//[^\n]*", "", open(path).read())
    word = r"(?:\w+(?:\.|->))?(?:tree_flags|seg_flags|status)\w*(?:\[[^\]]*\])?"
    stores = re.findall(r"(?<![\w*,(] )(?<!\w)\*\s*" + word + r"\s*=(?!=)", text)
    stores += re.findall(r"(?:seg_flags)\w*\[[^\]]*\]\s*=(?!=)", text)
    stores += re.findall(r"atomicExch\(\s*&?" + word, text)
    assert not stores
