"""Kernels that may start while the kernel before them on the stream still runs
(atm_stream.h): by their sources, each waits for it first, and no load can be
taken for one of memory that never changes and moved above the wait."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'atmosphere-model_b200', 'csrc')


def sources():
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, '*.cu')) + glob.glob(os.path.join(CSRC, '*.cuh'))):
        text = open(f).read()
        text = re.sub(r'//[^\n]*', '', text)
        out[os.path.basename(f)] = text
    return out


def kernels(text):
    """(name, parameters, body's beginning) of every kernel."""
    for m in re.finditer(r'__global__\s', text):
        end = text.index(') {', m.end())
        head = re.sub(r'__launch_bounds__\s*\([^{]*?\)\s*(?=k_)', '', text[m.end():end])
        name = re.search(r'\b(k_\w+)\s*\(', head)
        yield name.group(1), head[name.end():], text[end + 3:end + 400].lstrip()


def test_early_kernels_wait_first():
    src = sources()
    started = set()
    for text in src.values():
        started |= set(re.findall(r'\b(?:atm::)?launch\(\s*(k_\w+)', text))
        # kernels that a local function object launches for its caller
        if 'return launch(kernel' in text:
            started |= set(re.findall(r'\brun\((k_\w+)', text))
    assert len(started) > 25
    found = set()
    for name, text in src.items():
        for kernel, params, body in kernels(text):
            if kernel not in started:
                continue
            found.add(kernel)
            assert re.match(r'(atm::)?stream_order\(\);', body), (name, kernel)
            assert '__restrict__' not in params, (name, kernel)
    assert found >= started, started - found


def test_no_invariant_loads_behind_the_wait():
    for name, text in sources().items():
        if 'stream_order' not in text and 'column_at' not in text:
            continue
        for m in re.finditer(r'__ldg\(([^)]*)\)|ld\.global\.nc', text):
            assert m.group(1) and m.group(1).lstrip().startswith(('d_kap_', '(d_kap_')), (name, m.group(0))
