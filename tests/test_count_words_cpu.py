"""The facts the word count rests on (csrc/mc_words.cuh, word_tris), for all 256 rows of the case table."""
import os
import re

import daxtoolkit_gb300

TABLE = os.path.join(os.path.dirname(daxtoolkit_gb300.__file__), "csrc", "mc_tables.h")
#: The twelve edges, the faces as corner cycles and the opposite corners of a voxel.
EDGES = [(0, 1), (1, 2), (3, 2), (0, 3), (4, 5), (5, 6), (7, 6), (4, 7), (0, 4), (1, 5), (2, 6), (3, 7)]
FACES = [(0, 1, 2, 3), (4, 5, 6, 7), (0, 1, 5, 4), (3, 2, 6, 7), (0, 3, 7, 4), (1, 2, 6, 5)]
OPPOSITE = [(0, 6), (1, 7), (2, 4), (3, 5)]


def test_triangles_follow_from_the_edges_unless_a_face_or_two_corners_are_ambiguous():
    faces = [int(w, 16) >> 60 for w in re.findall(r"0x([0-9a-f]{16})ULL", open(TABLE).read())]
    assert len(faces) == 256
    looked_up = 0
    for case in range(256):
        def crosses(e):
            return (case >> e[0] & 1) != (case >> e[1] & 1)
        if case in (0, 255):
            assert faces[case] == 0
            continue
        ambiguous = any(all(crosses((f[n], f[(n + 1) % 4])) for n in range(4)) for f in FACES)
        cut_off = [all(crosses(e) for e in EDGES if v in e) for v in range(8)]
        if ambiguous or any(cut_off[a] and cut_off[b] for a, b in OPPOSITE):
            looked_up += 1
        else:
            assert faces[case] == sum(map(crosses, EDGES)) - 2, case
    assert looked_up == 128
