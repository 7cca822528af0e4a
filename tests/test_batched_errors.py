"""The batched engine's error word, read from the source: no wait of the persistent kernel can be
made to run out from outside, and its report must not depend on which iterations it ran out in."""
import os

from conftest import ROOT


def test_every_read_of_the_halt_words_looks_at_the_error_word():
    with open(os.path.join(ROOT, "itk_gb300", "csrc", "gb_batch.cu")) as f:
        source = f.read()
    # a run ends at its registrations' iteration limit: the last batch's words are read in collect_halted
    collect = source[source.index("static int collect_halted"):source.index('extern "C" int gb_batch_run')]
    run = source[source.index('extern "C" int gb_batch_run'):source.index('extern "C" int gb_batch_get_stats')]
    for text, words, first_use in ((collect, "b->h_halts", "b->h_halts[k]"), (run, "ph", "ph[n] == 0")):
        check = f"if ({words}[n + 1] != 0) return dependency_timeout();"
        assert check in text and text.index(check) < text.index(first_use)
