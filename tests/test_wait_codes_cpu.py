"""Every kernel file whose kernels wait with a limit reports a wait that ran out: it holds a pointer to
a word of host memory, stores a code there behind each such wait, and the backend hands it the word and
reads it. Nothing is made to run out here: the sources are read."""

import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bobcat_b200", "csrc")
WAITS = re.compile(r"\bmbar_(?:wait|test)\(")
SETTER = re.compile(r"cudaError_t (\w+_wait_word)\(int\* word\) \{ return cudaMemcpyToSymbol\(g_wait_word")


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def waiting_files():
    return [f for f in sorted(os.listdir(CSRC)) if f.endswith(".cu") and WAITS.search(source(f))]


def test_every_bounded_wait_reports():
    files = waiting_files()
    assert "kernels_matmul_few.cu" in files and len(files) >= 4
    backend = source("backend.cpp")
    for name in files:
        text = source(name)
        setter = SETTER.search(text)
        assert setter, "%s: a wait that runs out has nowhere to leave its code" % name
        assert "BC_CUDA(k::%s(words" % setter.group(1) in backend, "%s: the backend never hands it a word" % name
        assert re.search(r"\*reinterpret_cast<volatile int\*>\(g_wait_word\) = ", text), "%s: no wait stores a code" % name


def test_every_word_is_read():
    backend = source("backend.cpp")
    handed = re.findall(r"BC_CUDA\(k::\w+_wait_word\(words(?: \+ (\d+))?\)\)", backend)
    read = re.findall(r"= take\((\d+)\)", backend)
    words = int(re.search(r"kWaitWords = (\d+)", backend).group(1))
    assert sorted(int(i or 0) for i in handed) == sorted(int(i) for i in read) == list(range(words))


def test_the_few_row_kernel_tells_its_waits_apart():
    """On the copies of the weights and on the other warps' sums: the report names which one ran out."""
    calls = re.findall(r"wait_on\((\w+) [^;]*, (\d+)\);", source("kernels_matmul_few.cu"))
    assert sorted(calls) == [("bars", "1"), ("full_bars", "2")]
    assert re.search(r'gave up waiting for its %s \(code %d\)", code == 2 \? "weights" : "sums", code', source("backend.cpp"))
