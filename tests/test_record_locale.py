"""A foreign peer's tensor metadata is delivered as bytes whatever the process's locale: what counts as a letter in a
record's dtype name must not depend on it (in a single-byte locale byte 0xFF is a letter, and no UTF-8)."""
import os
import shutil
import subprocess
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
import ctypes, sys
sys.path.insert(0, sys.argv[1])
import torch
import tensorpipe_b200 as tpb
libc = ctypes.CDLL(None)
libc.setlocale.restype = ctypes.c_char_p
assert libc.setlocale(0, b"single_byte") == b"single_byte"
assert libc.isalnum(0xFF)
a, b = tpb.default_context("a", cuda=False), tpb.default_context("b", cuda=False)
listener = a.listen(["uv://127.0.0.1"])
accepted = listener.accept_future()
out_pipe = b.connect(listener.url("uv"))
in_pipe = accepted.result(30)
t, metadata = torch.randn(6), b'{"dtype": "\xff", "shape": [6]}'
coming = in_pipe.recv()
out_pipe.send([t], tensor_metadata=[metadata]).result(30)
got = coming.result(20)
assert got.tensor_metadata == [metadata] and got.tensors[0].dtype == torch.uint8
assert got.tensors[0].numpy().tobytes() == t.numpy().tobytes()
a.join(), b.join()
print("delivered")
"""


@pytest.mark.skipif(shutil.which("localedef") is None, reason="no localedef to make a locale with")
def test_bytes_beyond_ascii_in_a_single_byte_locale(built, tmp_path):
    charmap = ["<code_set_name> SINGLE-BYTE", "<comment_char> %", "<escape_char> /", "<mb_cur_min> 1", "<mb_cur_max> 1", "CHARMAP"]
    charmap += ["<U%04X> /x%02x c" % (i, i) for i in range(256)] + ["END CHARMAP", ""]
    (tmp_path / "charmap").write_text("\n".join(charmap))
    (tmp_path / "source").write_text("""comment_char %
escape_char /
LC_CTYPE
upper <U0041>..<U005A>
lower <U0061>..<U007A>;<U00FF>
alpha <U0041>..<U005A>;<U0061>..<U007A>;<U00FF>
digit <U0030>..<U0039>
space <U0009>..<U000D>;<U0020>
END LC_CTYPE
""")
    (tmp_path / "locales").mkdir()
    subprocess.run(["localedef", "-c", "--no-archive", "-f", "./charmap", "-i", "./source", "./locales/single_byte"],
                   cwd=tmp_path, capture_output=True)
    if not (tmp_path / "locales" / "single_byte" / "LC_CTYPE").exists():
        pytest.skip("localedef cannot make a locale here")
    env = dict(os.environ, LOCPATH=str(tmp_path / "locales"))
    out = subprocess.run([sys.executable, "-c", PROGRAM, REPO], env=env, capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and "delivered" in out.stdout, out.stdout + out.stderr
