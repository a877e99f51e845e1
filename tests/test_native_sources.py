"""What can be told of the native sources without compiling them or a GPU."""
import collections
import re


def test_every_exported_function_is_defined_once():
    """The library is linked from every source under the kernel folders: a second file with the same functions stops the link."""
    from openagents_b200 import _build
    for sources in (_build.cuda_sources(), _build.host_sources()):
        defined = collections.defaultdict(list)
        for path in sources:
            text = re.sub(r"//[^\n]*", "", path.read_text())
            for m in re.finditer(r"(?:B200_API|extern \"C\")[^;{}()]*?\b(b200_\w+)\s*\([^;{}]*\)\s*\{", text):
                defined[m.group(1)].append(path.name)
        assert len(defined) > 20
        assert {name: files for name, files in defined.items() if len(files) > 1} == {}
