// How far the synthesis beta pass (synth2.cuh) reads its table of d rows: a
// warp copies the rows of its (m, n) run in whole groups of four, so the last
// runs of the table, which are the shortest, reach past its last row.
#pragma once

constexpr int kRowGroup = 4;
// rows copied for a run of len rows
constexpr int rows_copied(int len) { return (len + kRowGroup - 1) / kRowGroup * kRowGroup; }
// rows allocated behind the last one: what a run of one row at the end reaches
constexpr int kRowPad = rows_copied(1) - 1;
