"""Events built pixel by pixel: FED payloads of the synthetic geometry's barrel layers 2 to 4 (the generator's
cabling: 24 modules per FED, two links per module, eight ROCs per link), for tests that need hits in given places."""
import struct

import numpy as np

MODULES_PER_FED = 24
LAYER_START = (0, 96, 320, 672)  # first module of barrel layers 1 to 4


def module(layer: int, ladder: int, z: int) -> int:
    """Module id of a barrel ladder's z-th module (0 to 7)."""
    return LAYER_START[layer - 1] + 8 * ladder + z


def word(mod: int, row: int, col: int, adc: int = 255) -> int:
    """The 32-bit payload word of a pixel (layers 2 to 4)."""
    assert LAYER_START[1] <= mod < 1184 and 0 <= row < 160 and 0 <= col < 416
    minus = mod % 8 < 4
    far = (row >= 80) == minus  # the half whose ROCs 8 to 15 read it
    if minus:
        roc, r, c = (8 + col // 52, 159 - row, col % 52) if far else (7 - col // 52, row, 51 - col % 52)
    else:
        roc, r, c = (15 - col // 52, row, 51 - col % 52) if far else (col // 52, 159 - row, col % 52)
    link = 2 * (mod % MODULES_PER_FED) + 1 + (roc >= 8)
    return (link << 26) | (((roc & 7) + 1) << 21) | ((c // 2) << 16) | ((2 * (80 - r) + c % 2) << 8) | adc


def event(pixels) -> bytes:
    """A raw event of (module, row, col) pixels; a module's words keep their order, which is the order of its hits."""
    feds = {}
    for mod, row, col in sorted(pixels, key=lambda p: p[0]):  # a stable sort
        feds.setdefault(mod // MODULES_PER_FED, []).append(word(mod, row, col))
    out = [struct.pack("<i", len(feds))]
    for f, words in sorted(feds.items()):
        words += [0] * (len(words) & 1)
        n64 = len(words) // 2 + 2
        out.append(struct.pack("<iiII", 1200 + f, 8 * n64, (1200 + f) << 8, 0x5 << 28))
        out.append(np.asarray(words, "<u4").tobytes() + struct.pack("<II", 0, (0xA << 28) | n64))
    return b"".join(out)


def batch(events):
    """(blob, offsets) of several events."""
    offs = np.concatenate([[0], np.cumsum([len(e) for e in events])]).astype(np.uint64)
    return np.frombuffer(b"".join(events), np.uint8), offs


# Two barrel ladders one behind the other (layer 2 ladder 7, layer 3 ladder 11), modules of z in 0 to 6.5 cm; an
# inner hit at row CENTRE + k looks at the outer ladder's rows around CENTRE + 1.6 k.
INNER, OUTER, CENTRE = module(2, 7, 4), module(3, 11, 4), 90


def grid(rows, cols):
    """Single-pixel clusters: rows and columns two apart."""
    return [(r, c) for c in cols for r in rows]
