// Groups of inherited face colours that are reduced together (dmc_mesh.cu, color_class): the group, 0..13, of
// colours 4..19 (LO) and 20..23 (HI), four bits each.
#pragma once
#define TMC_FRONT_GROUPS_LO 0x877654315432100dull
#define TMC_FRONT_GROUPS_HI 0xcba9ull
