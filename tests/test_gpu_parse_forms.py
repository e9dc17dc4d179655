"""The atom-line parser where its fast paths end: more than 19 digits, decimal exponents at +-40 and
beyond, halves between two numbers, lines too long for the staged copy, line starts at the edges of the
64-byte and 16 KB pieces; against Python's correctly rounded float()."""
import numpy as np
import pytest

from simulated_tem_gb300 import imaging

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    c = imaging.Context(0)
    yield c
    c.close()


NUMBERS = ["0", "-0.0", "+.5", "5.", "1e22", "1e23", "9007199254740993", "9007199254740993e0", "4503599627370497.5",
           "4503599627370496.5", "0.1", "123456789.0123456789", "12345678901234567890", "0.00000000000000000001234567",
           "1.7976931348623157e18", "3e-20", "1234567890123456789e-30", "1e-19", "8.5e20", "2.2250738585072011e-10",
           "9999999999999999999e-19", "1.00000000000000011102230246251565", "00000000000000000000012.50", "-7.25D+3", "6.02214076E23",
           "72057594037927945", "1.5d0", "1e+00000", "36893488147419103232e-5", "1e38", "4e-40", "1e-41"]


@pytest.mark.parametrize("n,pad", [(1, 0), (127, 0), (128, 3), (129, 70), (1500, 0), (700, 200), (40, 5000)])
def test_number_and_line_forms(ctx, n, pad):
    rng = np.random.default_rng(n)
    ids, lines, want = [], [], np.zeros((n, 3))
    for i in range(n):
        toks = [NUMBERS[int(j)] for j in rng.integers(0, len(NUMBERS), 3)]
        if i == 0:
            toks[1] = repr(rng.random())
        want[i] = [float(t.lower().replace("d", "e")) for t in toks]
        ty = int(rng.choice([1, 7, 123456789, 2147483647]))
        ids.append(ty)
        lines.append("%d\t%d %s,%s  %s" % (i + 1, ty, *toks) + " " * int(rng.integers(0, pad + 1)) + "\n")
    text = "".join(lines)
    if n % 2:
        text = text[:-1]  # the last line ends with the text
    b = torch.from_numpy(np.frombuffer(text.encode(), dtype=np.uint8).copy()).cuda()
    x = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    types = torch.zeros(n, dtype=torch.int32, device="cuda")
    bad = ctx.parse_atoms_device(b.data_ptr(), b.numel(), n, x.data_ptr(), types.data_ptr(),
                                 stream=torch.cuda.current_stream().cuda_stream)
    assert bad == -1
    got = x.cpu().numpy()
    assert np.array_equal(got, want) and np.array_equal(np.signbit(got), np.signbit(want))
    assert types.cpu().tolist() == ids


@pytest.mark.parametrize("line", ["7 1 1.0 2.0", "7 1 1.0 2.0 .", "7 1 1.0 2.0 1e", "7 x 1 2 3", "7 1 1 2 3x", "- 1 1 2 3",
                                  "7 1.0 1 2 3", "7 1 1.2.3 2 3", "7 1 1 2 --3"])
def test_malformed_lines(ctx, line):
    lines = ["%d 1 0.5 1.5 2.5" % (i + 1) for i in range(200)]
    lines[131] = line
    b = torch.from_numpy(np.frombuffer("\n".join(lines).encode(), dtype=np.uint8).copy()).cuda()
    x = torch.zeros((200, 3), dtype=torch.float64, device="cuda")
    assert ctx.parse_atoms_device(b.data_ptr(), b.numel(), 200, x.data_ptr(),
                                  stream=torch.cuda.current_stream().cuda_stream) == 131
