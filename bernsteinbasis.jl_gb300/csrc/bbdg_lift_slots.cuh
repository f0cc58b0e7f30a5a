// Generated by gen_lift_slots.py; do not edit. Entry q of a degree-N face stack lives at slot
// lift_slot<N>(q) (see the generator for how the slots were chosen).
#pragma once
#include <stdint.h>

template <int N>
__host__ __device__ __forceinline__ constexpr int lift_slot(int q) {
  return q;
}
// The same at run time, from device memory.
template <int N>
__device__ __forceinline__ int lift_slot_at(int q) {
  return q;
}

// N = 6: 14 wavefronts per element's gather (23 in volume order, 12 without conflicts)
template <>
__host__ __device__ __forceinline__ constexpr int lift_slot<6>(int q) {
  switch (q) {
    case 0: return 63; case 1: return 26; case 2: return 28; case 3: return 5;
    case 4: return 74; case 5: return 23; case 6: return 49; case 7: return 75;
    case 8: return 25; case 9: return 72; case 10: return 22; case 11: return 30;
    case 12: return 15; case 13: return 56; case 14: return 27; case 15: return 33;
    case 16: return 34; case 17: return 52; case 18: return 83; case 19: return 46;
    case 20: return 32; case 21: return 38; case 22: return 48; case 23: return 44;
    case 24: return 7; case 25: return 68; case 26: return 77; case 27: return 50;
    case 28: return 41; case 29: return 67; case 30: return 61; case 31: return 21;
    case 32: return 14; case 33: return 51; case 34: return 39; case 35: return 58;
    case 36: return 18; case 37: return 10; case 38: return 60; case 39: return 31;
    case 40: return 80; case 41: return 45; case 42: return 53; case 43: return 81;
    case 44: return 2; case 45: return 9; case 46: return 35; case 47: return 43;
    case 48: return 65; case 49: return 54; case 50: return 20; case 51: return 24;
    case 52: return 59; case 53: return 62; case 54: return 57; case 56: return 29;
    case 57: return 0; case 58: return 36; case 59: return 6; case 60: return 12;
    case 61: return 37; case 62: return 40; case 63: return 79; case 64: return 70;
    case 65: return 82; case 66: return 47; case 67: return 13; case 68: return 8;
    case 69: return 78; case 70: return 3; case 71: return 73; case 72: return 19;
    case 73: return 42; case 74: return 1; case 75: return 66; case 76: return 64;
    case 77: return 11; case 78: return 69; case 79: return 17; case 80: return 76;
    case 81: return 16; case 82: return 71; case 83: return 4;
    default: return q;
  }
}
static __device__ const uint16_t lift_slots_6[84] = {
    63, 26, 28, 5, 74, 23, 49, 75, 25, 72, 22, 30, 15, 56, 27, 33, 34, 52, 83, 46,
    32, 38, 48, 44, 7, 68, 77, 50, 41, 67, 61, 21, 14, 51, 39, 58, 18, 10, 60, 31,
    80, 45, 53, 81, 2, 9, 35, 43, 65, 54, 20, 24, 59, 62, 57, 55, 29, 0, 36, 6,
    12, 37, 40, 79, 70, 82, 47, 13, 8, 78, 3, 73, 19, 42, 1, 66, 64, 11, 69, 17,
    76, 16, 71, 4,
};
template <>
__device__ __forceinline__ int lift_slot_at<6>(int q) {
  return lift_slots_6[q];
}

// N = 7: 18 wavefronts per element's gather (42 in volume order, 16 without conflicts)
template <>
__host__ __device__ __forceinline__ constexpr int lift_slot<7>(int q) {
  switch (q) {
    case 0: return 55; case 1: return 60; case 2: return 81; case 3: return 117;
    case 4: return 57; case 5: return 47; case 6: return 86; case 7: return 99;
    case 8: return 45; case 9: return 40; case 10: return 30; case 11: return 36;
    case 12: return 90; case 13: return 24; case 14: return 59; case 15: return 83;
    case 16: return 31; case 17: return 105; case 18: return 32; case 19: return 71;
    case 20: return 108; case 21: return 93; case 22: return 66; case 23: return 78;
    case 24: return 82; case 25: return 38; case 26: return 5; case 27: return 10;
    case 28: return 1; case 29: return 116; case 30: return 43; case 31: return 48;
    case 32: return 3; case 33: return 119; case 34: return 111; case 35: return 8;
    case 36: return 75; case 37: return 12; case 38: return 88; case 39: return 97;
    case 40: return 62; case 41: return 63; case 42: return 84; case 43: return 29;
    case 44: return 50; case 45: return 34; case 46: return 6; case 47: return 0;
    case 48: return 14; case 49: return 89; case 50: return 91; case 51: return 42;
    case 52: return 58; case 53: return 37; case 54: return 112; case 55: return 21;
    case 56: return 92; case 57: return 77; case 58: return 68; case 59: return 7;
    case 60: return 49; case 61: return 19; case 62: return 22; case 63: return 9;
    case 64: return 26; case 65: return 51; case 66: return 114; case 67: return 104;
    case 68: return 61; case 69: return 15; case 70: return 103; case 71: return 95;
    case 72: return 28; case 73: return 65; case 74: return 106; case 75: return 100;
    case 76: return 67; case 77: return 113; case 78: return 56; case 79: return 94;
    case 80: return 20; case 81: return 110; case 82: return 44; case 83: return 98;
    case 84: return 96; case 85: return 73; case 86: return 109; case 87: return 70;
    case 88: return 101; case 89: return 27; case 90: return 25; case 91: return 80;
    case 92: return 107; case 93: return 85; case 94: return 54; case 95: return 23;
    case 96: return 33; case 97: return 18; case 98: return 102; case 99: return 53;
    case 100: return 39; case 101: return 74; case 102: return 46; case 103: return 16;
    case 104: return 41; case 105: return 87; case 106: return 17; case 107: return 79;
    case 108: return 72; case 109: return 13; case 110: return 64; case 111: return 2;
    case 112: return 4; case 113: return 115; case 114: return 69; case 115: return 11;
    case 116: return 52; case 117: return 118; case 118: return 76; case 119: return 35;
    default: return q;
  }
}
static __device__ const uint16_t lift_slots_7[120] = {
    55, 60, 81, 117, 57, 47, 86, 99, 45, 40, 30, 36, 90, 24, 59, 83, 31, 105, 32, 71,
    108, 93, 66, 78, 82, 38, 5, 10, 1, 116, 43, 48, 3, 119, 111, 8, 75, 12, 88, 97,
    62, 63, 84, 29, 50, 34, 6, 0, 14, 89, 91, 42, 58, 37, 112, 21, 92, 77, 68, 7,
    49, 19, 22, 9, 26, 51, 114, 104, 61, 15, 103, 95, 28, 65, 106, 100, 67, 113, 56, 94,
    20, 110, 44, 98, 96, 73, 109, 70, 101, 27, 25, 80, 107, 85, 54, 23, 33, 18, 102, 53,
    39, 74, 46, 16, 41, 87, 17, 79, 72, 13, 64, 2, 4, 115, 69, 11, 52, 118, 76, 35,
};
template <>
__device__ __forceinline__ int lift_slot_at<7>(int q) {
  return lift_slots_7[q];
}

// N = 8: 29 wavefronts per element's gather (56 in volume order, 24 without conflicts)
template <>
__host__ __device__ __forceinline__ constexpr int lift_slot<8>(int q) {
  switch (q) {
    case 0: return 37; case 1: return 120; case 2: return 23; case 3: return 43;
    case 4: return 63; case 5: return 65; case 6: return 70; case 7: return 163;
    case 8: return 155; case 9: return 92; case 10: return 32; case 11: return 78;
    case 12: return 58; case 13: return 79; case 14: return 89; case 15: return 84;
    case 16: return 48; case 17: return 81; case 18: return 125; case 19: return 72;
    case 20: return 149; case 21: return 45; case 22: return 51; case 23: return 62;
    case 24: return 73; case 25: return 71; case 26: return 34; case 27: return 76;
    case 28: return 118; case 29: return 42; case 30: return 146; case 31: return 164;
    case 32: return 101; case 33: return 47; case 34: return 21; case 35: return 49;
    case 36: return 27; case 37: return 121; case 38: return 112; case 39: return 102;
    case 40: return 137; case 41: return 67; case 42: return 162; case 43: return 0;
    case 44: return 100; case 45: return 109; case 47: return 104; case 48: return 116;
    case 49: return 90; case 50: return 103; case 51: return 157; case 52: return 94;
    case 53: return 18; case 54: return 83; case 55: return 150; case 56: return 74;
    case 57: return 139; case 58: return 12; case 59: return 55; case 60: return 161;
    case 61: return 124; case 62: return 152; case 63: return 95; case 64: return 128;
    case 65: return 114; case 66: return 144; case 67: return 61; case 68: return 97;
    case 69: return 123; case 70: return 54; case 71: return 148; case 72: return 39;
    case 73: return 19; case 74: return 30; case 75: return 159; case 76: return 87;
    case 77: return 14; case 78: return 28; case 79: return 154; case 80: return 1;
    case 81: return 44; case 82: return 143; case 83: return 153; case 84: return 138;
    case 85: return 68; case 86: return 113; case 87: return 66; case 88: return 56;
    case 89: return 8; case 90: return 141; case 91: return 69; case 92: return 131;
    case 93: return 134; case 94: return 130; case 95: return 105; case 96: return 26;
    case 97: return 38; case 98: return 52; case 99: return 5; case 100: return 25;
    case 101: return 142; case 102: return 111; case 103: return 33; case 104: return 96;
    case 105: return 98; case 106: return 77; case 107: return 88; case 108: return 99;
    case 109: return 22; case 110: return 156; case 111: return 50; case 112: return 115;
    case 113: return 117; case 114: return 41; case 115: return 108; case 116: return 10;
    case 117: return 16; case 118: return 91; case 119: return 135; case 120: return 127;
    case 121: return 158; case 122: return 40; case 123: return 107; case 124: return 132;
    case 125: return 119; case 126: return 17; case 127: return 29; case 128: return 11;
    case 129: return 136; case 130: return 64; case 131: return 80; case 132: return 145;
    case 133: return 59; case 134: return 31; case 135: return 133; case 136: return 20;
    case 137: return 86; case 138: return 36; case 139: return 147; case 140: return 82;
    case 141: return 24; case 142: return 3; case 143: return 60; case 144: return 140;
    case 145: return 9; case 146: return 93; case 147: return 7; case 148: return 6;
    case 149: return 151; case 150: return 15; case 151: return 110; case 152: return 13;
    case 153: return 85; case 154: return 106; case 155: return 126; case 156: return 2;
    case 157: return 129; case 158: return 122; case 159: return 57; case 161: return 35;
    case 162: return 4; case 163: return 75; case 164: return 53;
    default: return q;
  }
}
static __device__ const uint16_t lift_slots_8[165] = {
    37, 120, 23, 43, 63, 65, 70, 163, 155, 92, 32, 78, 58, 79, 89, 84, 48, 81, 125, 72,
    149, 45, 51, 62, 73, 71, 34, 76, 118, 42, 146, 164, 101, 47, 21, 49, 27, 121, 112, 102,
    137, 67, 162, 0, 100, 109, 46, 104, 116, 90, 103, 157, 94, 18, 83, 150, 74, 139, 12, 55,
    161, 124, 152, 95, 128, 114, 144, 61, 97, 123, 54, 148, 39, 19, 30, 159, 87, 14, 28, 154,
    1, 44, 143, 153, 138, 68, 113, 66, 56, 8, 141, 69, 131, 134, 130, 105, 26, 38, 52, 5,
    25, 142, 111, 33, 96, 98, 77, 88, 99, 22, 156, 50, 115, 117, 41, 108, 10, 16, 91, 135,
    127, 158, 40, 107, 132, 119, 17, 29, 11, 136, 64, 80, 145, 59, 31, 133, 20, 86, 36, 147,
    82, 24, 3, 60, 140, 9, 93, 7, 6, 151, 15, 110, 13, 85, 106, 126, 2, 129, 122, 57,
    160, 35, 4, 75, 53,
};
template <>
__device__ __forceinline__ int lift_slot_at<8>(int q) {
  return lift_slots_8[q];
}

// N = 9: 32 wavefronts per element's gather (70 in volume order, 28 without conflicts)
template <>
__host__ __device__ __forceinline__ constexpr int lift_slot<9>(int q) {
  switch (q) {
    case 0: return 178; case 1: return 99; case 2: return 180; case 3: return 150;
    case 4: return 58; case 5: return 171; case 6: return 23; case 7: return 33;
    case 8: return 158; case 9: return 45; case 10: return 166; case 11: return 101;
    case 12: return 189; case 13: return 46; case 14: return 201; case 15: return 63;
    case 16: return 47; case 17: return 108; case 18: return 147; case 19: return 170;
    case 20: return 104; case 21: return 217; case 22: return 162; case 23: return 81;
    case 24: return 0; case 25: return 181; case 26: return 164; case 27: return 167;
    case 28: return 219; case 29: return 208; case 30: return 24; case 31: return 92;
    case 32: return 212; case 33: return 127; case 34: return 39; case 35: return 109;
    case 36: return 30; case 37: return 69; case 38: return 157; case 39: return 134;
    case 40: return 203; case 41: return 60; case 42: return 210; case 43: return 91;
    case 44: return 130; case 45: return 131; case 46: return 118; case 47: return 129;
    case 48: return 44; case 49: return 87; case 50: return 179; case 51: return 32;
    case 52: return 218; case 53: return 78; case 54: return 56; case 55: return 36;
    case 56: return 169; case 57: return 143; case 58: return 17; case 59: return 25;
    case 60: return 106; case 61: return 85; case 62: return 168; case 63: return 80;
    case 64: return 159; case 65: return 200; case 66: return 128; case 67: return 68;
    case 68: return 126; case 69: return 156; case 70: return 121; case 71: return 27;
    case 72: return 13; case 73: return 55; case 74: return 52; case 75: return 110;
    case 76: return 114; case 77: return 154; case 78: return 6; case 79: return 19;
    case 80: return 209; case 81: return 125; case 82: return 75; case 83: return 98;
    case 84: return 41; case 85: return 120; case 86: return 74; case 87: return 35;
    case 88: return 214; case 89: return 204; case 90: return 97; case 91: return 111;
    case 92: return 197; case 93: return 149; case 94: return 7; case 95: return 144;
    case 96: return 141; case 97: return 113; case 98: return 196; case 99: return 105;
    case 100: return 31; case 101: return 198; case 102: return 187; case 103: return 172;
    case 104: return 28; case 105: return 152; case 106: return 64; case 107: return 103;
    case 108: return 51; case 109: return 82; case 110: return 66; case 111: return 202;
    case 112: return 116; case 113: return 215; case 114: return 207; case 115: return 29;
    case 116: return 43; case 117: return 193; case 118: return 16; case 119: return 37;
    case 120: return 86; case 121: return 174; case 122: return 163; case 123: return 62;
    case 124: return 136; case 125: return 153; case 126: return 53; case 127: return 90;
    case 128: return 49; case 129: return 4; case 130: return 18; case 131: return 89;
    case 132: return 148; case 133: return 102; case 134: return 139; case 135: return 72;
    case 136: return 206; case 137: return 5; case 138: return 83; case 139: return 93;
    case 140: return 34; case 141: return 3; case 142: return 155; case 143: return 73;
    case 144: return 22; case 145: return 26; case 146: return 1; case 147: return 213;
    case 148: return 173; case 149: return 190; case 150: return 124; case 151: return 216;
    case 152: return 199; case 153: return 95; case 154: return 42; case 155: return 119;
    case 156: return 76; case 157: return 175; case 158: return 96; case 159: return 48;
    case 160: return 115; case 161: return 59; case 162: return 15; case 163: return 138;
    case 164: return 183; case 165: return 185; case 166: return 176; case 167: return 188;
    case 168: return 100; case 169: return 84; case 170: return 61; case 171: return 184;
    case 172: return 38; case 173: return 135; case 174: return 107; case 175: return 195;
    case 176: return 9; case 177: return 192; case 178: return 182; case 179: return 205;
    case 180: return 161; case 181: return 191; case 182: return 40; case 183: return 14;
    case 184: return 194; case 185: return 21; case 186: return 94; case 187: return 122;
    case 188: return 177; case 189: return 50; case 190: return 165; case 191: return 140;
    case 192: return 112; case 193: return 67; case 194: return 146; case 195: return 117;
    case 196: return 186; case 197: return 20; case 198: return 137; case 199: return 151;
    case 200: return 11; case 201: return 88; case 202: return 77; case 203: return 54;
    case 204: return 142; case 205: return 145; case 206: return 123; case 207: return 133;
    case 208: return 70; case 209: return 57; case 210: return 2; case 211: return 10;
    case 212: return 65; case 213: return 12; case 214: return 211; case 215: return 132;
    case 216: return 8; case 217: return 71; case 218: return 79; case 219: return 160;
    default: return q;
  }
}
static __device__ const uint16_t lift_slots_9[220] = {
    178, 99, 180, 150, 58, 171, 23, 33, 158, 45, 166, 101, 189, 46, 201, 63, 47, 108, 147, 170,
    104, 217, 162, 81, 0, 181, 164, 167, 219, 208, 24, 92, 212, 127, 39, 109, 30, 69, 157, 134,
    203, 60, 210, 91, 130, 131, 118, 129, 44, 87, 179, 32, 218, 78, 56, 36, 169, 143, 17, 25,
    106, 85, 168, 80, 159, 200, 128, 68, 126, 156, 121, 27, 13, 55, 52, 110, 114, 154, 6, 19,
    209, 125, 75, 98, 41, 120, 74, 35, 214, 204, 97, 111, 197, 149, 7, 144, 141, 113, 196, 105,
    31, 198, 187, 172, 28, 152, 64, 103, 51, 82, 66, 202, 116, 215, 207, 29, 43, 193, 16, 37,
    86, 174, 163, 62, 136, 153, 53, 90, 49, 4, 18, 89, 148, 102, 139, 72, 206, 5, 83, 93,
    34, 3, 155, 73, 22, 26, 1, 213, 173, 190, 124, 216, 199, 95, 42, 119, 76, 175, 96, 48,
    115, 59, 15, 138, 183, 185, 176, 188, 100, 84, 61, 184, 38, 135, 107, 195, 9, 192, 182, 205,
    161, 191, 40, 14, 194, 21, 94, 122, 177, 50, 165, 140, 112, 67, 146, 117, 186, 20, 137, 151,
    11, 88, 77, 54, 142, 145, 123, 133, 70, 57, 2, 10, 65, 12, 211, 132, 8, 71, 79, 160,
};
template <>
__device__ __forceinline__ int lift_slot_at<9>(int q) {
  return lift_slots_9[q];
}

// N = 11: 57 wavefronts per element's gather (123 in volume order, 48 without conflicts)
template <>
__host__ __device__ __forceinline__ constexpr int lift_slot<11>(int q) {
  switch (q) {
    case 0: return 217; case 1: return 45; case 2: return 90; case 3: return 98;
    case 4: return 240; case 5: return 165; case 6: return 100; case 7: return 175;
    case 8: return 138; case 9: return 343; case 10: return 50; case 11: return 33;
    case 12: return 142; case 13: return 232; case 14: return 102; case 15: return 182;
    case 16: return 105; case 17: return 123; case 18: return 7; case 19: return 220;
    case 20: return 127; case 21: return 116; case 22: return 331; case 23: return 285;
    case 24: return 158; case 25: return 177; case 26: return 184; case 27: return 320;
    case 28: return 309; case 29: return 108; case 30: return 243; case 31: return 163;
    case 32: return 313; case 33: return 272; case 34: return 347; case 35: return 284;
    case 36: return 325; case 37: return 215; case 38: return 305; case 39: return 270;
    case 40: return 265; case 41: return 212; case 42: return 268; case 43: return 359;
    case 44: return 13; case 45: return 66; case 46: return 218; case 47: return 278;
    case 48: return 126; case 49: return 287; case 50: return 356; case 51: return 19;
    case 52: return 326; case 53: return 306; case 54: return 289; case 55: return 43;
    case 56: return 111; case 57: return 42; case 58: return 152; case 59: return 253;
    case 60: return 72; case 61: return 195; case 62: return 96; case 63: return 149;
    case 64: return 31; case 65: return 206; case 66: return 15; case 67: return 242;
    case 68: return 122; case 69: return 339; case 70: return 151; case 71: return 353;
    case 72: return 71; case 73: return 226; case 74: return 323; case 75: return 234;
    case 76: return 201; case 77: return 296; case 78: return 84; case 79: return 224;
    case 80: return 86; case 81: return 28; case 82: return 203; case 83: return 187;
    case 84: return 358; case 85: return 209; case 86: return 300; case 87: return 56;
    case 88: return 117; case 89: return 357; case 90: return 141; case 91: return 61;
    case 92: return 48; case 93: return 89; case 94: return 62; case 95: return 36;
    case 96: return 118; case 97: return 110; case 98: return 101; case 99: return 303;
    case 100: return 225; case 101: return 41; case 102: return 147; case 103: return 362;
    case 104: return 146; case 105: return 20; case 106: return 88; case 107: return 159;
    case 108: return 327; case 109: return 294; case 110: return 136; case 111: return 363;
    case 112: return 160; case 113: return 53; case 114: return 292; case 115: return 237;
    case 116: return 251; case 117: return 60; case 118: return 29; case 119: return 144;
    case 120: return 355; case 121: return 236; case 122: return 113; case 123: return 57;
    case 124: return 94; case 125: return 290; case 126: return 183; case 127: return 186;
    case 128: return 199; case 129: return 69; case 130: return 54; case 131: return 12;
    case 132: return 233; case 133: return 269; case 134: return 249; case 135: return 316;
    case 136: return 91; case 137: return 273; case 138: return 16; case 139: return 330;
    case 140: return 68; case 141: return 192; case 142: return 198; case 143: return 139;
    case 144: return 73; case 145: return 334; case 146: return 350; case 147: return 95;
    case 148: return 231; case 149: return 349; case 150: return 40; case 151: return 307;
    case 152: return 131; case 153: return 162; case 154: return 314; case 155: return 164;
    case 156: return 79; case 157: return 193; case 158: return 338; case 159: return 148;
    case 160: return 23; case 161: return 304; case 162: return 38; case 163: return 17;
    case 164: return 35; case 165: return 132; case 166: return 150; case 167: return 262;
    case 168: return 293; case 169: return 301; case 170: return 190; case 171: return 354;
    case 172: return 154; case 173: return 221; case 174: return 275; case 175: return 47;
    case 176: return 97; case 177: return 82; case 178: return 351; case 179: return 202;
    case 180: return 277; case 181: return 8; case 182: return 216; case 183: return 288;
    case 184: return 235; case 185: return 14; case 186: return 155; case 187: return 188;
    case 188: return 180; case 189: return 281; case 190: return 361; case 191: return 103;
    case 192: return 166; case 193: return 2; case 194: return 267; case 195: return 222;
    case 196: return 197; case 197: return 196; case 198: return 37; case 199: return 120;
    case 200: return 135; case 201: return 259; case 202: return 181; case 203: return 87;
    case 204: return 129; case 205: return 25; case 206: return 308; case 207: return 352;
    case 208: return 315; case 209: return 137; case 210: return 10; case 211: return 115;
    case 212: return 49; case 213: return 255; case 214: return 109; case 215: return 264;
    case 216: return 0; case 217: return 18; case 218: return 78; case 219: return 207;
    case 220: return 92; case 221: return 317; case 222: return 140; case 223: return 246;
    case 224: return 77; case 225: return 256; case 226: return 153; case 227: return 248;
    case 228: return 70; case 229: return 282; case 230: return 322; case 231: return 9;
    case 232: return 283; case 233: return 311; case 234: return 210; case 235: return 208;
    case 236: return 213; case 237: return 145; case 238: return 227; case 239: return 104;
    case 240: return 125; case 241: return 276; case 242: return 214; case 243: return 65;
    case 244: return 261; case 245: return 260; case 246: return 223; case 247: return 172;
    case 248: return 106; case 249: return 238; case 250: return 51; case 251: return 239;
    case 252: return 167; case 253: return 30; case 254: return 124; case 255: return 171;
    case 256: return 32; case 257: return 245; case 258: return 194; case 259: return 58;
    case 260: return 179; case 261: return 336; case 262: return 263; case 263: return 59;
    case 264: return 119; case 265: return 74; case 266: return 178; case 267: return 257;
    case 268: return 360; case 269: return 67; case 270: return 286; case 271: return 156;
    case 272: return 302; case 273: return 133; case 274: return 271; case 275: return 228;
    case 276: return 191; case 277: return 332; case 278: return 333; case 279: return 344;
    case 280: return 189; case 281: return 230; case 282: return 75; case 283: return 310;
    case 284: return 52; case 285: return 297; case 286: return 337; case 287: return 345;
    case 288: return 93; case 289: return 312; case 290: return 204; case 292: return 219;
    case 293: return 329; case 294: return 341; case 295: return 121; case 296: return 34;
    case 297: return 11; case 298: return 335; case 299: return 4; case 300: return 241;
    case 301: return 229; case 302: return 342; case 303: return 295; case 304: return 340;
    case 305: return 1; case 306: return 211; case 307: return 64; case 308: return 328;
    case 309: return 176; case 310: return 348; case 311: return 173; case 312: return 318;
    case 313: return 114; case 314: return 134; case 315: return 319; case 316: return 174;
    case 317: return 279; case 318: return 26; case 319: return 170; case 320: return 321;
    case 321: return 168; case 322: return 250; case 323: return 107; case 324: return 85;
    case 325: return 46; case 326: return 157; case 327: return 298; case 328: return 6;
    case 329: return 27; case 330: return 143; case 331: return 274; case 332: return 128;
    case 333: return 99; case 334: return 22; case 335: return 324; case 336: return 5;
    case 337: return 130; case 338: return 185; case 339: return 254; case 340: return 63;
    case 341: return 244; case 342: return 169; case 343: return 80; case 344: return 81;
    case 345: return 247; case 346: return 83; case 347: return 280; case 348: return 252;
    case 349: return 205; case 350: return 39; case 351: return 44; case 352: return 3;
    case 353: return 55; case 354: return 161; case 355: return 266; case 356: return 346;
    case 357: return 112; case 358: return 200; case 359: return 24; case 360: return 21;
    case 361: return 258; case 362: return 299; case 363: return 76;
    default: return q;
  }
}
static __device__ const uint16_t lift_slots_11[364] = {
    217, 45, 90, 98, 240, 165, 100, 175, 138, 343, 50, 33, 142, 232, 102, 182, 105, 123, 7, 220,
    127, 116, 331, 285, 158, 177, 184, 320, 309, 108, 243, 163, 313, 272, 347, 284, 325, 215, 305, 270,
    265, 212, 268, 359, 13, 66, 218, 278, 126, 287, 356, 19, 326, 306, 289, 43, 111, 42, 152, 253,
    72, 195, 96, 149, 31, 206, 15, 242, 122, 339, 151, 353, 71, 226, 323, 234, 201, 296, 84, 224,
    86, 28, 203, 187, 358, 209, 300, 56, 117, 357, 141, 61, 48, 89, 62, 36, 118, 110, 101, 303,
    225, 41, 147, 362, 146, 20, 88, 159, 327, 294, 136, 363, 160, 53, 292, 237, 251, 60, 29, 144,
    355, 236, 113, 57, 94, 290, 183, 186, 199, 69, 54, 12, 233, 269, 249, 316, 91, 273, 16, 330,
    68, 192, 198, 139, 73, 334, 350, 95, 231, 349, 40, 307, 131, 162, 314, 164, 79, 193, 338, 148,
    23, 304, 38, 17, 35, 132, 150, 262, 293, 301, 190, 354, 154, 221, 275, 47, 97, 82, 351, 202,
    277, 8, 216, 288, 235, 14, 155, 188, 180, 281, 361, 103, 166, 2, 267, 222, 197, 196, 37, 120,
    135, 259, 181, 87, 129, 25, 308, 352, 315, 137, 10, 115, 49, 255, 109, 264, 0, 18, 78, 207,
    92, 317, 140, 246, 77, 256, 153, 248, 70, 282, 322, 9, 283, 311, 210, 208, 213, 145, 227, 104,
    125, 276, 214, 65, 261, 260, 223, 172, 106, 238, 51, 239, 167, 30, 124, 171, 32, 245, 194, 58,
    179, 336, 263, 59, 119, 74, 178, 257, 360, 67, 286, 156, 302, 133, 271, 228, 191, 332, 333, 344,
    189, 230, 75, 310, 52, 297, 337, 345, 93, 312, 204, 291, 219, 329, 341, 121, 34, 11, 335, 4,
    241, 229, 342, 295, 340, 1, 211, 64, 328, 176, 348, 173, 318, 114, 134, 319, 174, 279, 26, 170,
    321, 168, 250, 107, 85, 46, 157, 298, 6, 27, 143, 274, 128, 99, 22, 324, 5, 130, 185, 254,
    63, 244, 169, 80, 81, 247, 83, 280, 252, 205, 39, 44, 3, 55, 161, 266, 346, 112, 200, 24,
    21, 258, 299, 76,
};
template <>
__device__ __forceinline__ int lift_slot_at<11>(int q) {
  return lift_slots_11[q];
}
